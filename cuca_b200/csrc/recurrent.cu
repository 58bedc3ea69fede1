// Recurrent mixers: state carried from token to token in 32-bit, one slot per request.
//   mingru_scan        S = (1 - z) S + z c, gates from the current token alone
//   causal_conv        short convolution per channel over a request's tokens, its last inputs kept per request
//   ssm_scan           S = exp(-exp(A) dt) S + dt B x^T, y = S^T C + D x per head (scalar decay per head)
//   gated_group_norm   y * silu(z), RMS-normed in equal parts, times a weight
// A step brings each request a run of consecutive rows (req_row0, req_count); a kernel walks a request's rows in
// order from the state its slot holds and leaves the new state there. The order of the arithmetic along a sequence
// does not depend on where it was cut into steps, but for the state-space scan's long portions in segments (16-bit models).
#include "common.cuh"
#include "state_rows.cuh"
#include <math.h>

namespace {

__device__ __forceinline__ float sigmoidf_(float v) { return 1.f / (1.f + expf(-v)); }
__device__ __forceinline__ float siluf_(float v) { return v / (1.f + expf(-v)); }

// zxg: [rows, 3 W] 32-bit (z, u and g before their activations, biases added). One thread per (request, channel).
template <typename TO>
__global__ void mingru_scan_kernel(const float* __restrict__ zxg, float* __restrict__ state, TO* __restrict__ out,
                                   const int* __restrict__ req_row0, const int* __restrict__ req_count,
                                   const int* __restrict__ slots, int W) {
  pdl_trigger();
  pdl_wait();
  const int q = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int slot = slots[q], n = req_count[q], r0 = req_row0[q];
  if (slot < 0 || n <= 0 || c >= W) return;
  float S = state[(size_t)slot * W + c];
  // eight tokens' inputs are requested before the first is used: the chain through S is short, the loads are not
  constexpr int U = 8;
  for (int t0 = 0; t0 < n; t0 += U) {
    float zr[U], ur[U], gr[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (t0 + i < n) {
        const float* row = zxg + (size_t)(r0 + t0 + i) * 3 * W;
        zr[i] = row[c]; ur[i] = row[W + c]; gr[i] = row[2 * W + c];
      }
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (t0 + i < n) {
        const float z = sigmoidf_(zr[i]);
        const float u = ur[i];
        const float cand = u >= 0.f ? u + 0.5f : sigmoidf_(u);
        S = (1.f - z) * S + z * cand;
        out[(size_t)(r0 + t0 + i) * W + c] = from_f32<TO>(S * siluf_(gr[i]));
      }
    }
  }
  state[(size_t)slot * W + c] = S;
}

// The same recurrence over long portions, cut into chunks of L tokens that run side by side: S_t = a_t S_(t-1) + b_t
// with a = 1 - z, b = z c composes, so a chunk is summed up as (product of a, its own end state from zero), the
// chunks' start states follow from those in one short pass per channel, and every chunk then runs from its start
// state. phase 0: chunk sums into carry[q][k][0..1][c]; phase 1: start states into carry[q][k][0][c], the request's
// state brought up to date; phase 2: the outputs. The start states are rounded differently than token by token.
template <typename TO>
__global__ void mingru_chunked_kernel(const float* __restrict__ zxg, float* __restrict__ state, float* __restrict__ carry,
                                      TO* __restrict__ out, const int* __restrict__ req_row0,
                                      const int* __restrict__ req_count, const int* __restrict__ slots, int W, int L,
                                      int max_chunks, int phase) {
  pdl_trigger();
  pdl_wait();
  const int q = blockIdx.z, k = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int slot = slots[q], n = req_count[q], r0 = req_row0[q];
  if (slot < 0 || n <= 0 || c >= W) return;
  const int n_chunks = (n + L - 1) / L;
  float* cq = carry + (size_t)q * max_chunks * 2 * W;
  if (phase == 1) {
    float S = state[(size_t)slot * W + c];
    for (int j = 0; j < n_chunks; ++j) {
      const float a = cq[(size_t)(2 * j) * W + c], b = cq[(size_t)(2 * j + 1) * W + c];
      cq[(size_t)(2 * j) * W + c] = S;
      S = fmaf(a, S, b);
    }
    state[(size_t)slot * W + c] = S;
    return;
  }
  if (k >= n_chunks) return;
  const int t1 = (k + 1) * L < n ? (k + 1) * L : n;
  float a = 1.f, S = phase == 0 ? 0.f : cq[(size_t)(2 * k) * W + c];
  for (int t = k * L; t < t1; ++t) {
    const float* row = zxg + (size_t)(r0 + t) * 3 * W;
    const float z = sigmoidf_(row[c]);
    const float u = row[W + c];
    const float cand = u >= 0.f ? u + 0.5f : sigmoidf_(u);
    S = (1.f - z) * S + z * cand;
    if (phase == 0) a *= 1.f - z;
    else out[(size_t)(r0 + t) * W + c] = from_f32<TO>(S * siluf_(row[2 * W + c]));
  }
  if (phase == 0) {
    cq[(size_t)(2 * k) * W + c] = a;
    cq[(size_t)(2 * k + 1) * W + c] = S;
  }
}

// in: 32-bit rows of stride ld_in, channel c at column col0 + c. kept: [slots, taps - 1, C] the inputs before the
// request's first row of this step (zeros for a new request). Rows that have taps - 1 rows of their own request before
// them in this step are plain rows; a request's first taps - 1 rows and then its new kept inputs are one block's work
// (only that block touches them): channel c of request q.
template <typename TW>
__device__ __forceinline__ void conv_request(const float* __restrict__ in, int ld_in, int col0, const TW* __restrict__ wc, float b0,
                                             float* __restrict__ kept, float* __restrict__ out, const int* __restrict__ req_row0,
                                             const int* __restrict__ req_count, const int* __restrict__ slots, int C, int taps,
                                             int c, int q) {
  const int back = taps - 1;
  if (back == 0) return;  // a one-tap convolution keeps nothing and every row was a plain row
  const int slot = slots[q], n = req_count[q], r0 = req_row0[q];
  if (slot < 0 || n <= 0) return;
  float* keep = kept + (size_t)slot * back * C;
  // val(m): the input m rows after the request's first row of this step; m < 0 reaches into the kept inputs
  auto val = [&](int m) -> float {
    return m < 0 ? keep[(size_t)(m + back) * C + c] : in[(size_t)(r0 + m) * ld_in + col0 + c];
  };
  const int head = n < back ? n : back;
  for (int j = 0; j < head; ++j) {
    float acc = b0;
    for (int k = 0; k < taps; ++k) acc = fmaf(to_f32(wc[k]), val(j - back + k), acc);
    out[(size_t)(r0 + j) * C + c] = siluf_(acc);
  }
  // new kept inputs: the last `back` inputs of the sequence so far. Ascending k reads entries at or after the one
  // it writes (old entry n + k for the new entry k), so nothing is overwritten before it is read.
  for (int k = 0; k < back; ++k) {
    const float v = val(n - back + k);
    keep[(size_t)k * C + c] = v;
  }
}

// A row a thread: blocks y < n_rows take a row each, blocks y >= n_rows a request each.
template <typename TW>
__global__ void causal_conv_kernel(const float* __restrict__ in, int ld_in, int col0, const TW* __restrict__ w,
                                   const TW* __restrict__ bias, float* __restrict__ kept, float* __restrict__ out,
                                   const int* __restrict__ seq_of_row, const int* __restrict__ req_row0,
                                   const int* __restrict__ req_count, const int* __restrict__ slots, int n_rows,
                                   int C, int taps) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int b = blockIdx.y;
  const int back = taps - 1;
  const TW* wc = w + (size_t)c * taps;
  const float b0 = bias ? to_f32(bias[c]) : 0.f;
  if (b < n_rows) {
    const int seq = seq_of_row[b];
    if (seq < 0 || b < back || (back > 0 && seq_of_row[b - back] != seq)) return;
    float acc = b0;
    for (int k = 0; k < taps; ++k)
      acc = fmaf(to_f32(wc[k]), in[(size_t)(b - back + k) * ld_in + col0 + c], acc);
    out[(size_t)b * C + c] = siluf_(acc);
    return;
  }
  conv_request(in, ld_in, col0, wc, b0, kept, out, req_row0, req_count, slots, C, taps, c, b - n_rows);
}

// CONV_ROWS rows a thread. TAPS: taps known at compile time (a thread then reads every input of its rows once, all of them
// in flight together), or 0.
constexpr int CONV_ROWS = 16;
template <typename TW, int TAPS>
__global__ void causal_conv_many_kernel(const float* __restrict__ in, int ld_in, int col0, const TW* __restrict__ w,
                                        const TW* __restrict__ bias, float* __restrict__ kept, float* __restrict__ out,
                                        const int* __restrict__ seq_of_row, const int* __restrict__ req_row0,
                                        const int* __restrict__ req_count, const int* __restrict__ slots, int n_rows,
                                        int C, int taps) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int row_blocks = (n_rows + CONV_ROWS - 1) / CONV_ROWS;
  const int back = (TAPS ? TAPS : taps) - 1;
  const TW* wc = w + (size_t)c * (back + 1);
  const float b0 = bias ? to_f32(bias[c]) : 0.f;
  if ((int)blockIdx.y >= row_blocks) {
    conv_request(in, ld_in, col0, wc, b0, kept, out, req_row0, req_count, slots, C, taps, c, (int)blockIdx.y - row_blocks);
    return;
  }
  const int r0 = blockIdx.y * CONV_ROWS, r1 = min(n_rows, r0 + CONV_ROWS);
  auto whole = [&](int b) {  // whether row b has `back` rows of its request before it
    const int seq = b < r1 ? seq_of_row[b] : -1;
    return seq >= 0 && b >= back && (back == 0 || seq_of_row[b - back] == seq);
  };
  if (TAPS) {
    float taps_w[TAPS ? TAPS : 1], x[CONV_ROWS + (TAPS ? TAPS : 1) - 1];
#pragma unroll
    for (int k = 0; k < TAPS; ++k) taps_w[k] = to_f32(wc[k]);
#pragma unroll
    for (int i = 0; i < CONV_ROWS + TAPS - 1; ++i) {
      const int b = r0 - (TAPS - 1) + i;
      x[i] = b >= 0 && b < r1 ? in[(size_t)b * ld_in + col0 + c] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < CONV_ROWS; ++i) {
      if (!whole(r0 + i)) continue;
      float acc = b0;
#pragma unroll
      for (int k = 0; k < TAPS; ++k) acc = fmaf(taps_w[k], x[i + k], acc);
      out[(size_t)(r0 + i) * C + c] = siluf_(acc);
    }
  } else {
    for (int b = r0; b < r1; ++b) {
      if (!whole(b)) continue;
      float acc = b0;
      for (int k = 0; k <= back; ++k) acc = fmaf(to_f32(wc[k]), in[(size_t)(b - back + k) * ld_in + col0 + c], acc);
      out[(size_t)b * C + c] = siluf_(acc);
    }
  }
}

constexpr int SSM_MAX_STATE = 1024;
constexpr int SSM_SEGMENT = 512;  // tokens of a segment (below)
constexpr int SSM_MAX_CUT = 64;

// The requests of a step whose portions are cut: request q[i], ascending, has the cells first[i] .. first[i + 1] - 1, one a segment.
struct Cut {
  int n;
  int q[SSM_MAX_CUT], first[SSM_MAX_CUT + 1];
};

// One block per (head, request, run of PB value columns); a column's state rows lie with NS threads (see Split).
// state: [slots, H, P, N]. xbc: 32-bit [rows, H P + 2 G N] after the convolution (x | B | C); dt_raw: rows of stride
// ld_dt, head h at column dt_col + h, before bias and softplus.
// Tokens hang together through one multiply-add per state value alone, so the kernel is bound by how many instructions
// it issues and by its reads of shared memory: eight rows of four columns a thread, pairs of rows in every instruction.
// CUT: blocks of segments come first, each from no state but the request's first, whose state goes to its cell (see
// ssm_join_kernel), then those of the requests that are walked whole.
template <typename S_, bool CUT>
__global__ void __launch_bounds__(128)
ssm_scan_kernel(const float* __restrict__ xbc, const float* __restrict__ dt_raw, int ld_dt, int dt_col,
                const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                const float* __restrict__ d_skip, float* __restrict__ state, float* __restrict__ y,
                const int* __restrict__ req_row0, const int* __restrict__ req_count,
                const int* __restrict__ slots, int H, int P, int N, int G, int wide, float* __restrict__ ends,
                float* __restrict__ decays, const __grid_constant__ Cut cut) {
  constexpr int NS = S_::NS, NC = S_::NC, DP = S_::DP, PB = S_::PB, TC = S_::TC, PAIRS = S_::PAIRS;
  constexpr int PER = 2 * DP + ((PB + 1 + 3) & ~3);  // a token: B, C, the block's x, the raw step size
  static_assert(TC <= 32, "a lane a token");
  extern __shared__ __align__(16) float sm[];
  __shared__ float steps[4][TC][2];  // a warp's own: step size, decay
  pdl_trigger();
  pdl_wait();
  int h = blockIdx.x, q = blockIdx.y, seg = 0, unit = 0;
  bool segment = false;
  if (CUT) {
    h = blockIdx.x % H;
    unit = blockIdx.x / H;
    segment = unit < cut.first[cut.n];
    int i = 0;
    if (segment) {
      while (unit >= cut.first[i + 1]) ++i;
      q = cut.q[i];
      seg = unit - cut.first[i];
    } else {
      q = unit - cut.first[cut.n];
      while (i < cut.n && cut.q[i] <= q) ++i, ++q;
    }
  }
  const int slot = slots[q], whole = req_count[q], n = segment ? min(SSM_SEGMENT, whole - seg * SSM_SEGMENT) : whole;
  const int r0 = req_row0[q] + seg * SSM_SEGMENT;
  if (slot < 0 || n <= 0) return;
  const int lane = threadIdx.x & 31;
  const int col_local = threadIdx.x / NS, s = threadIdx.x % NS;
  const int col0 = blockIdx.z * PB, at = col_local * NC;
  const int cols = min(NC, P - col0 - at);              // columns of this thread that exist (none: 0 or less)
  const int g = h / (H / G);
  const int C = H * P + 2 * G * N;
  float* st = state + (((size_t)slot * H + h) * P + (cols > 0 ? col0 + at : 0)) * N;
  f32x2 S[NC][PAIRS];
  load_rows<S_>(S, st, s, N, seg > 0 ? 0 : cols, wide);
  const size_t cell = (size_t)unit * H + h;
  if (segment) st = ends + (cell * P + (cols > 0 ? col0 + at : 0)) * N;
  float product = 1.f;  // of the decays
  const float A = -expf(a_log[h]);
  const float bias = dt_bias[h], D = d_skip[h];
  // what no copy writes: rows from N on (B = C = 0) and the values of columns from P on
  {
    const int spare = DP - N, there = min(PB, P - col0), fill = 2 * spare + PB - there;
    for (int e = threadIdx.x; e < (n < TC ? n : 2 * TC) * fill; e += 128) {
      const int t = e / fill, w = e % fill;
      float* tok = sm + t * PER;
      if (w < 2 * spare) tok[(w / spare) * DP + N + w % spare] = 0.f;
      else tok[2 * DP + there + (w - 2 * spare)] = 0.f;
    }
  }
  __syncthreads();
  // Two runs of TC tokens: the next run's copies (cp.async) are in flight while this one is worked through.
  auto stage = [&](int t0, int buf) {
    const int nt = n - t0 < TC ? n - t0 : TC;
    float* base = sm + buf * TC * PER;
    auto copy = [&](int t, int which, int r) {
      const float* src = xbc + (size_t)(r0 + t0 + t) * C + H * P + (which * G + g) * N + r;
      if (r < N) cp_async_f(base + t * PER + which * DP + r, src, wide);
    };
    if (wide)
      for (int e = threadIdx.x; e < nt * 2 * (DP / 4); e += 128) copy(e / (2 * (DP / 4)), e / (DP / 4) % 2, e % (DP / 4) * 4);
    else
      for (int e = threadIdx.x; e < nt * 2 * DP; e += 128) copy(e / (2 * DP), e / DP % 2, e % DP);
    for (int e = threadIdx.x; e < nt * PB; e += 128) {
      const int t = e / PB, i = e % PB;
      if (col0 + i < P) cp_async_f(base + t * PER + 2 * DP + i, xbc + (size_t)(r0 + t0 + t) * C + h * P + col0 + i, false);
    }
    if (threadIdx.x < nt)
      cp_async_f(base + threadIdx.x * PER + 2 * DP + PB, dt_raw + (size_t)(r0 + t0 + threadIdx.x) * ld_dt + dt_col + h, false);
    cp_async_commit();
  };
  float(*mine)[2] = steps[threadIdx.x >> 5];
  const int n_chunks = (n + TC - 1) / TC;
  stage(0, 0);
  for (int c = 0; c < n_chunks; ++c) {
    if (c + 1 < n_chunks) { stage((c + 1) * TC, (c + 1) & 1); cp_async_wait<1>(); }
    else cp_async_wait<0>();
    __syncthreads();
    const int t0 = c * TC, nt = n - t0 < TC ? n - t0 : TC;
    const float* tok = sm + (c & 1) * TC * PER;
    if (lane < nt) {  // step size and decay of every token of the run
      const float raw = tok[lane * PER + 2 * DP + PB] + bias;
      const float dt = raw > 20.f ? raw : log1pf(expf(raw));
      mine[lane][0] = dt;
      mine[lane][1] = expf(A * dt);
    }
    __syncwarp();
    float* y_at = y + (size_t)(r0 + t0) * (H * P) + h * P + col0 + at;
    // several tokens at once, their outputs summed together: thread s writes value s / (NS / (count NC)) of
    // [tokens][columns]
    auto walk = [&](int t, auto count) {
      constexpr int U = decltype(count)::value;
      const float* first = tok;
      float acc[U * NC];
#pragma unroll
      for (int i = 0; i < U; ++i, tok += PER) {
        f32x2 B[PAIRS], Cv[PAIRS];
        float x[NC];
        staged_rows<S_>(B, tok, s);
        staged_rows<S_>(Cv, tok + DP, s);
        staged_values<NC>(x, tok + 2 * DP, at);
        const float dt = mine[t + i][0];
        const f32x2 decay = f2_both(mine[t + i][1]);
        if (CUT) product *= mine[t + i][1];
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const f32x2 dx = f2_both(dt * x[j]);
#pragma unroll
          for (int e = 0; e < PAIRS; ++e) S[j][e] = f2_fma(decay, S[j][e], f2_mul(dx, B[e]));
          acc[i * NC + j] = dot_rows(S[j], Cv);
        }
      }
      constexpr int LANES = NS / (U * NC);
      const float sum = spread_sum<NS, U * NC>(acc, s);
      const int own = s / LANES;
      if (s % LANES == 0 && own % NC < cols)
        y_at[(size_t)(t + own / NC) * (H * P) + own % NC] = sum + D * first[(own / NC) * PER + 2 * DP + at + own % NC];
    };
    int t = 0;
    for (; t + S_::U <= nt; t += S_::U) walk(t, Count<S_::U>());
    for (; t < nt; ++t) walk(t, Count<1>());
    __syncthreads();  // this run is read to the end before the run after next is copied over it
  }
  store_rows<S_>(S, st, s, N, cols, wide);
  if (segment && threadIdx.x == 0 && blockIdx.z == 0) decays[cell] = product;
}

// What a segment's tokens owe to the segments before it. A prompt's scan is 2,048 steps one behind the other in a warp a
// scheduler, so it is cut into segments that run side by side, each from no state; with S the state a segment should have
// begun with, its outputs lack C_t S times the decays since, and the state behind it lacks S times all of its decays.
// One block per (head, segment behind a request's first, JOIN of its tokens): S from the segments' ends in turn, then 64
// tokens x 64 columns at a time as a contraction in 32 bits, 4 x 4 outputs a thread, bound by shared memory. 64 heads of
// 64 x 128, 2,048 tokens in four segments: scan 340 -> 218 us and 80 for this. Requests of one segment are scanned as before.
constexpr int JOIN = 256, JOIN_P = 64, JOIN_PITCH = JOIN_P + 4;
// a state's share behind a decay that may have come out as zero: what is no number stays so, as it does token by token
__device__ __forceinline__ float decayed(float d, float v) { return d > 0.f ? d * v : (fabsf(v) <= 3.402823466e38f ? 0.f : v); }
__global__ void __launch_bounds__(256)
ssm_join_kernel(const float* __restrict__ xbc, const float* __restrict__ dt_raw, int ld_dt, int dt_col,
                const float* __restrict__ dt_bias, const float* __restrict__ a_log, float* __restrict__ state,
                float* __restrict__ y, const int* __restrict__ req_row0, const int* __restrict__ req_count,
                const int* __restrict__ slots, int H, int P, int N, int G, const float* __restrict__ ends,
                const float* __restrict__ decays, const __grid_constant__ Cut cut) {
  extern __shared__ __align__(16) float sm[];
  float* S = sm;                        // [N][JOIN_PITCH]
  float* Cs = S + N * JOIN_PITCH;       // [64][N + 4]
  float* since = Cs + 64 * (N + 4);     // [SSM_SEGMENT]: the decays of the segment up to and with each token
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, tid = threadIdx.x, part0 = blockIdx.z * JOIN;
  int i = 0;
  while ((int)blockIdx.y >= cut.first[i + 1] - (i + 1)) ++i;  // (each request before has a first segment that is not joined)
  const int q = cut.q[i], seg = 1 + blockIdx.y - (cut.first[i] - i), cell0 = cut.first[i];
  const int slot = slots[q], whole = req_count[q], n = min(SSM_SEGMENT, whole - seg * SSM_SEGMENT);
  if (slot < 0 || n <= part0) return;
  const int g = h / (H / G), C = H * P + 2 * G * N, row0 = req_row0[q] + seg * SSM_SEGMENT;
  const bool last = part0 == 0 && (seg + 1) * SSM_SEGMENT >= whole;  // this block leaves the request's state behind
  auto cell = [&](int k) { return (size_t)(cell0 + k) * H + h; };
  for (int e = tid; e < P * N; e += 256) {
    float v = ends[cell(0) * P * N + e];
    for (int k = 1; k < seg; ++k) v = decayed(decays[cell(k)], v) + ends[cell(k) * P * N + e];
    S[e % N * JOIN_PITCH + e / N] = v;
    if (last) state[((size_t)slot * H + h) * P * N + e] = decayed(decays[cell(seg)], v) + ends[cell(seg) * P * N + e];
  }
  for (int e = tid; e < N * (JOIN_P - P); e += 256) S[e / (JOIN_P - P) * JOIN_PITCH + P + e % (JOIN_P - P)] = 0.f;
  const int end = min(n, part0 + JOIN);
  const float A = -expf(a_log[h]), bias = dt_bias[h];
  for (int t = tid; t < end; t += 256) {
    const float raw = dt_raw[(size_t)(row0 + t) * ld_dt + dt_col + h] + bias;
    since[t] = expf(A * (raw > 20.f ? raw : log1pf(expf(raw))));
  }
  __syncthreads();
  if (tid < 32) {  // products up to each token: a run of 16 a lane, then over the lanes
    constexpr int RUN = SSM_SEGMENT / 32;
    float p = 1.f;
    for (int i = 0; i < RUN; ++i) {
      const int t = tid * RUN + i;
      if (t < end) since[t] = p *= since[t];
    }
    float before = p;
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, before, o);
      if (tid >= o) before *= v;
    }
    before = __shfl_up_sync(0xffffffffu, before, 1);
    if (tid > 0)
      for (int i = 0; i < RUN; ++i)
        if (tid * RUN + i < end) since[tid * RUN + i] *= before;
  }
  const int tx = tid % 16, ty = tid / 16;
  for (int t0 = part0; t0 < end; t0 += 64) {
    __syncthreads();  // (the products are there; the tile before is read)
    for (int e = tid; e < 64 * (N / 4); e += 256) {
      const int t = e / (N / 4), k = e % (N / 4) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t0 + t < end) v = *reinterpret_cast<const float4*>(xbc + (size_t)(row0 + t0 + t) * C + H * P + (G + g) * N + k);
      *reinterpret_cast<float4*>(Cs + t * (N + 4) + k) = v;
    }
    __syncthreads();
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 2
    for (int k = 0; k < N; k += 4) {
      float4 c[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) c[i] = *reinterpret_cast<const float4*>(Cs + (ty + 16 * i) * (N + 4) + k);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 b = *reinterpret_cast<const float4*>(S + (k + u) * JOIN_PITCH + 4 * tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float cu = u == 0 ? c[i].x : u == 1 ? c[i].y : u == 2 ? c[i].z : c[i].w;
          acc[i][0] = fmaf(cu, b.x, acc[i][0]);
          acc[i][1] = fmaf(cu, b.y, acc[i][1]);
          acc[i][2] = fmaf(cu, b.z, acc[i][2]);
          acc[i][3] = fmaf(cu, b.w, acc[i][3]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = t0 + ty + 16 * i;
      if (t >= end || 4 * tx >= P) continue;
      float4* at = reinterpret_cast<float4*>(y + (size_t)(row0 + t) * (H * P) + h * P + 4 * tx);
      float4 v = *at;
      const float d = since[t];
      v.x += decayed(d, acc[i][0]);
      v.y += decayed(d, acc[i][1]);
      v.z += decayed(d, acc[i][2]);
      v.w += decayed(d, acc[i][3]);
      *at = v;
    }
  }
}

// One block per (row, part). v = y * silu(z); out = v * rsqrt(mean over the part (v^2) + eps) * w.
template <typename TW, typename TO>
__global__ void __launch_bounds__(256)
gated_group_norm_kernel(const float* __restrict__ y, const float* __restrict__ z, int ld_z, const TW* __restrict__ w,
                        TO* __restrict__ out, int inner, int part, float eps) {
  __shared__ float red[8];
  pdl_trigger();
  pdl_wait();
  const size_t row = blockIdx.y;
  const int c0 = blockIdx.x * part;
  float s = 0.f;
  // parts of up to 4096 values stay in registers between the two passes (all loads of the row in flight together)
  constexpr int KEEP = 16;
  float kept[KEEP];
  const bool keep = part <= KEEP * 256;
  if (keep) {
    float yv[KEEP], zv[KEEP];
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
      const int i = threadIdx.x + k * 256;
      if (i < part) { yv[k] = y[row * inner + c0 + i]; zv[k] = z[row * ld_z + c0 + i]; }
    }
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
      const int i = threadIdx.x + k * 256;
      kept[k] = i < part ? yv[k] * siluf_(zv[k]) : 0.f;
      s = fmaf(kept[k], kept[k], s);
    }
  } else {
    for (int i = threadIdx.x; i < part; i += 256) {
      const float v = y[row * inner + c0 + i] * siluf_(z[row * ld_z + c0 + i]);
      s = fmaf(v, v, s);
    }
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float inv = rsqrtf(tot / (float)part + eps);
  if (keep) {
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
      const int i = threadIdx.x + k * 256;
      if (i < part) out[row * inner + c0 + i] = from_f32<TO>(kept[k] * inv * to_f32(w[c0 + i]));
    }
    return;
  }
  for (int i = threadIdx.x; i < part; i += 256) {
    const float v = y[row * inner + c0 + i] * siluf_(z[row * ld_z + c0 + i]);
    out[row * inner + c0 + i] = from_f32<TO>(v * inv * to_f32(w[c0 + i]));
  }
}

}  // namespace

CUCA_API int cuca_mingru_scan(const float* zxg, float* state, void* out, int out_dtype, const int* req_row0,
                              const int* req_count, const int* slots, int n_seqs, int W, cudaStream_t stream) {
  if (n_seqs == 0) return 0;
  CUCA_REQUIRE(W > 0 && n_seqs <= 65535, "mingru_scan: bad sizes W=%d requests=%d", W, n_seqs);
  dim3 grid((W + 127) / 128, n_seqs);
  if (out_dtype == CUCA_F32)
    cuca_launch(mingru_scan_kernel<float>, grid, dim3(128), 0, stream, true, zxg, state, (float*)out, req_row0,
                req_count, slots, W);
  else if (out_dtype == CUCA_BF16)
    cuca_launch(mingru_scan_kernel<__nv_bfloat16>, grid, dim3(128), 0, stream, true, zxg, state, (__nv_bfloat16*)out,
                req_row0, req_count, slots, W);
  else
    CUCA_REQUIRE(false, "mingru_scan: unknown dtype %d", out_dtype);
  CUCA_CHECK_LAUNCH("mingru_scan");
  return 0;
}

// Long portions in chunks of `L` tokens side by side (see the kernel). carry: [n_seqs, max_chunks, 2, W] 32-bit
// scratch, max_chunks >= ceil(longest portion / L).
CUCA_API int cuca_mingru_scan_chunked(const float* zxg, float* state, float* carry, void* out, int out_dtype,
                                      const int* req_row0, const int* req_count, const int* slots, int n_seqs, int W,
                                      int L, int max_chunks, cudaStream_t stream) {
  if (n_seqs == 0) return 0;
  CUCA_REQUIRE(W > 0 && L > 0 && max_chunks > 0 && n_seqs <= 65535 && max_chunks <= 65535,
               "mingru_scan_chunked: bad sizes W=%d L=%d chunks=%d requests=%d", W, L, max_chunks, n_seqs);
  for (int phase = 0; phase < 3; ++phase) {
    dim3 grid((W + 127) / 128, phase == 1 ? 1 : max_chunks, n_seqs);
    if (out_dtype == CUCA_F32)
      cuca_launch(mingru_chunked_kernel<float>, grid, dim3(128), 0, stream, true, zxg, state, carry, (float*)out,
                  req_row0, req_count, slots, W, L, max_chunks, phase);
    else if (out_dtype == CUCA_BF16)
      cuca_launch(mingru_chunked_kernel<__nv_bfloat16>, grid, dim3(128), 0, stream, true, zxg, state, carry,
                  (__nv_bfloat16*)out, req_row0, req_count, slots, W, L, max_chunks, phase);
    else
      CUCA_REQUIRE(false, "mingru_scan_chunked: unknown dtype %d", out_dtype);
    CUCA_CHECK_LAUNCH("mingru_scan_chunked");
  }
  return 0;
}

CUCA_API int cuca_causal_conv(const float* in, int ld_in, int col0, const void* w, const void* bias, int w_dtype,
                              float* kept, float* out, const int* seq_of_row, const int* req_row0,
                              const int* req_count, const int* slots, int n_rows, int n_seqs, int C, int taps,
                              cudaStream_t stream) {
  if (n_rows == 0) return 0;
  CUCA_REQUIRE(C > 0 && taps >= 1, "causal_conv: bad sizes channels=%d taps=%d", C, taps);
  CUCA_REQUIRE(n_rows + n_seqs <= 65535, "causal_conv: %d rows in one step exceed the launch limit", n_rows);
  // 16 rows a thread read every input once, but pay only where their blocks fill the GPU: measured with four taps, us a row a
  // thread, 16 rows: 2,048 x 4,352 (4,352 blocks) 75, 22; 200 x 4,352 (442) 8.8, 5.7; 40 x 4,352 (102) 3.7, 4.2; 1,501 x 100
  // (94) 3.3, 4.3; other numbers of taps (a loop, one load after the other): 1,501 x 4,352, three taps 53, 26; 2,400 x 768
  // (900) 15.8, 17.5; 200 x 4,352 7.9, 9.7.
  const long long blocks = (long long)((C + 127) / 128) * ((n_rows + CONV_ROWS - 1) / CONV_ROWS);
  const bool many = blocks >= (taps == 4 ? 2 : 8) * cuca_device_sms();
  const dim3 grid((C + 127) / 128, (many ? (n_rows + CONV_ROWS - 1) / CONV_ROWS : n_rows) + n_seqs);
#define CONV(KERNEL, TW)                                                                                              \
  cuca_launch(KERNEL, grid, dim3(128), 0, stream, true, in, ld_in, col0, (const TW*)w, (const TW*)bias, kept, out,    \
              seq_of_row, req_row0, req_count, slots, n_rows, C, taps)
#define CONV_OF(TW)                                                       \
  do {                                                                    \
    if (!many) CONV(causal_conv_kernel<TW>, TW);                          \
    else if (taps == 4) CONV((causal_conv_many_kernel<TW, 4>), TW);       \
    else CONV((causal_conv_many_kernel<TW, 0>), TW);                      \
  } while (0)
  if (w_dtype == CUCA_F32) CONV_OF(float);
  else if (w_dtype == CUCA_BF16) CONV_OF(__nv_bfloat16);
  else CUCA_REQUIRE(false, "causal_conv: unknown dtype %d", w_dtype);
#undef CONV_OF
#undef CONV
  CUCA_CHECK_LAUNCH("causal_conv");
  return 0;
}

// Tokens of a segment, and whether the sizes allow segments.
CUCA_API int cuca_ssm_segment() { return SSM_SEGMENT; }
CUCA_API int cuca_ssm_segments_allowed(int P, int N) { return P > 0 && P <= JOIN_P && P % 4 == 0 && N > 0 && N <= 128 && N % 4 == 0; }

// Calls `go` with the split of the state that its size takes.
template <typename F>
static int with_split(int N, F go) {
  // Few state values a column: threads of four rows, so that a block's columns are no more than a head has (64). Measured
  // with eight and four rows a thread, us: 80 heads of 64 x 16, 1,501 tokens 365, 205, 256 requests of a token 77, 48; 24
  // heads of 64 x 64, 1,501 tokens 344, 197, 64 prompts of 40 52, 58 (as at 64 x 128: 249, 296, so eight rows stay there).
  if (N <= 16) return go(Split<4, 4, 2>());
  if (N <= 32) return go(Split<8, 4, 4>());
  if (N <= 64) return go(Split<16, 4, 4>());
  if (N <= 128) return go(Split<16, 8, 4>());
  if (N <= 256) return go(Split<32, 8, 4>());
  if (N <= 512) return go(Split<32, 16, 4>());
  return go(Split<32, 32, 2>());
}

// The portions that are cut where one of at least `cut_from` tokens is: requests of counts[0 .. n_seqs - 1] tokens.
static Cut cut_of(const int* counts, int n_seqs, int cut_from) {
  Cut cut = {};
  for (int q = 0; q < n_seqs && cut.n < SSM_MAX_CUT; ++q) {
    if (counts[q] < cut_from || counts[q] <= SSM_SEGMENT) continue;
    cut.q[cut.n] = q;
    cut.first[cut.n + 1] = cut.first[cut.n] + (counts[q] + SSM_SEGMENT - 1) / SSM_SEGMENT;
    ++cut.n;
  }
  return cut;
}

// Cells that cuca_ssm_scan's scratch has to hold: one a segment, whatever other requests the step has.
CUCA_API int cuca_ssm_cells(const int* counts, int n_seqs, int cut_from) {
  const Cut cut = cut_of(counts, n_seqs, cut_from);
  return cut.first[cut.n];
}

// From how many tokens on a step's portions are better off cut, 0: none. Segments pay where a whole walk leaves an SM one block
// at most or little more, which it keeps waiting for one step after the other; blocks that share an SM fill each other's waits,
// and then the join is all that segments bring. Measured, us (whole, cut): 64 heads of 64 x 128 (128 blocks a request) 1,024 tokens
// 172, 200, 2,048 340, 304, four requests of 2,048 864, 1,010; 80 heads 2,048 494, 389; 128 heads 493, 524. 24 heads of 64 x 64,
// 600 tokens 81, 103, 1,024 136, 114, 2,048 269, 136, eight requests of 1,100 246, 327; 64 heads of 64 x 16, 600 tokens 84, 80,
// 1,024 140, 90, eight requests of 1,100 234, 307.
CUCA_API int cuca_ssm_cut_from(const int* counts, int n_seqs, int H, int P, int N) {
  if (!cuca_ssm_segments_allowed(P, N)) return 0;
  const int from = N > 64 ? 3 * SSM_SEGMENT : 2 * SSM_SEGMENT;
  long long n = 0;
  for (int q = 0; q < n_seqs; ++q) n += counts[q] >= from;
  const int columns = with_split(N, [](auto split) { return (int)decltype(split)::PB; });
  const long long blocks = n * H * ((P + columns - 1) / columns);
  return n > 0 && n <= SSM_MAX_CUT && 4 * blocks <= 5ll * cuca_device_sms() ? from : 0;
}

// cut_from > 0: portions of at least so many tokens and more than cuca_ssm_segment() (the first 64 of them) have their segments
// walked side by side (another rounding). counts: the requests' tokens, as in req_count, on the host; scratch: cuca_ssm_cells
// times H (P N + 1) floats, 16-byte aligned.
CUCA_API int cuca_ssm_scan(const float* xbc, const float* dt_raw, int ld_dt, int dt_col, const float* dt_bias,
                           const float* a_log, const float* d_skip, float* state, float* y, const int* req_row0,
                           const int* req_count, const int* slots, int n_seqs, int H, int P, int N, int G, int cut_from,
                           const int* counts, float* scratch, cudaStream_t stream) {
  if (n_seqs == 0) return 0;
  CUCA_REQUIRE(H > 0 && P > 0 && N > 0 && G > 0 && H % G == 0, "ssm_scan: bad sizes heads=%d vdim=%d state=%d groups=%d",
               H, P, N, G);
  CUCA_REQUIRE(n_seqs <= 65535, "ssm_scan: %d requests exceed the launch limit", n_seqs);
  CUCA_REQUIRE(N <= SSM_MAX_STATE, "ssm_scan: state size %d exceeds %d", N, SSM_MAX_STATE);
  const int wide = N % 4 == 0 && (H * P) % 4 == 0 && (((uintptr_t)xbc | (uintptr_t)state) & 15) == 0;
  const Cut cut = cut_from > 0 && counts ? cut_of(counts, n_seqs, cut_from) : Cut{};
  const int cells = cut.first[cut.n], units = cells + n_seqs - cut.n;
  CUCA_REQUIRE(!cut.n || (cuca_ssm_segments_allowed(P, N) && scratch &&
                          (((uintptr_t)xbc | (uintptr_t)state | (uintptr_t)y | (uintptr_t)scratch) & 15) == 0 && (H * P + 2 * G * N) % 4 == 0 &&
                          cells <= 65535 && (long long)H * units < (1ll << 31)), "ssm_scan: %d segments of %d x %d", cells, P, N);
  float* ends = scratch;
  float* decays = scratch + (size_t)cells * H * P * N;
  const int rc = with_split(N, [&](auto split) {
    using C = decltype(split);
    const int per_token = 2 * C::DP + ((C::PB + 4) & ~3);
    if (cut.n)
      return launch_scan<C>("ssm_scan", ssm_scan_kernel<C, true>, per_token, H * units, 1, P, stream, xbc, dt_raw, ld_dt, dt_col, dt_bias,
                            a_log, d_skip, state, y, req_row0, req_count, slots, H, P, N, G, wide, ends, decays, cut);
    return launch_scan<C>("ssm_scan", ssm_scan_kernel<C, false>, per_token, H, n_seqs, P, stream, xbc, dt_raw, ld_dt, dt_col, dt_bias,
                          a_log, d_skip, state, y, req_row0, req_count, slots, H, P, N, G, wide, ends, decays, cut);
  });
  if (rc || !cut.n) return rc;
  const int smem = (N * JOIN_PITCH + 64 * (N + 4) + SSM_SEGMENT) * 4;
  static const cudaError_t e = cudaFuncSetAttribute(ssm_join_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (128 * JOIN_PITCH + 64 * 132 + SSM_SEGMENT) * 4);
  CUCA_REQUIRE(e == cudaSuccess, "ssm_scan: %d bytes of shared memory were refused: %s", smem, cudaGetErrorString(e));
  cuca_launch(ssm_join_kernel, dim3(H, cells - cut.n, SSM_SEGMENT / JOIN), dim3(256), smem, stream, true, xbc, dt_raw, ld_dt, dt_col,
              dt_bias, a_log, state, y, req_row0, req_count, slots, H, P, N, G, (const float*)ends, (const float*)decays, cut);
  CUCA_CHECK_LAUNCH("ssm_join");
  return 0;
}

CUCA_API int cuca_gated_group_norm(const float* y, const float* z, int ld_z, const void* w, int w_dtype, void* out,
                                   int out_dtype, int n_rows, int inner, int parts, float eps, cudaStream_t stream) {
  if (n_rows == 0) return 0;
  CUCA_REQUIRE(parts > 0 && inner % parts == 0, "gated_group_norm: %d parts do not divide %d", parts, inner);
  CUCA_REQUIRE(n_rows <= 65535, "gated_group_norm: %d rows exceed the launch limit", n_rows);
  dim3 grid(parts, n_rows);
  const int part = inner / parts;
#define GGN(TW, TO)                                                                                               \
  cuca_launch(gated_group_norm_kernel<TW, TO>, grid, dim3(256), 0, stream, true, y, z, ld_z, (const TW*)w, (TO*)out, \
              inner, part, eps)
  if (w_dtype == CUCA_F32 && out_dtype == CUCA_F32) GGN(float, float);
  else if (w_dtype == CUCA_BF16 && out_dtype == CUCA_BF16) GGN(__nv_bfloat16, __nv_bfloat16);
  else if (w_dtype == CUCA_F32 && out_dtype == CUCA_BF16) GGN(float, __nv_bfloat16);
  else CUCA_REQUIRE(false, "gated_group_norm: unsupported dtypes %d/%d", w_dtype, out_dtype);
#undef GGN
  CUCA_CHECK_LAUNCH("gated_group_norm");
  return 0;
}
