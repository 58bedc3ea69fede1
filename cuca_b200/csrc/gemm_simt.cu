// Plain CUDA-core contraction out = A[M,K] * W[N,K]^T with 32-bit accumulation:
// the true 32-bit path of every projection, and the bfloat16 path's stand-in
// for shapes the tensor-core kernel refuses. Each output element is summed in one
// order whatever M and the kernel's form are, so a row's result never depends on
// the rest of the batch: the K products of a run of CHUNK in ascending order with
// fused multiply-adds from zero, and the runs' sums in ascending order.
//
// Two forms. Up to FEW rows, and a few more over narrow outputs (`rows_kernel`): a block takes 16 weight rows and all of K
// and a thread one run of one row for all tokens, so that the reading of the weights is what bounds it. Above
// (`tile_kernel`): register tiles of 8 x 8 or 4 x 8 outputs a thread, bound by the multiply-adds (128 a clock and SM).
// Both read 16 bytes at a time with asynchronous copies where sizes and addresses allow it (32-bit operands,
// K and the row stride multiples of 4); otherwise through registers (the tile form two elements at a time where K, the row
// stride and the addresses are even), with the same arithmetic.
//
// Measured on the Llama-3.2-1B widths in 32-bit: 4 rows, SwiGLU of 2 x 8192 x 2048 40 us (3.4 TB/s of weights), head of
// 32,000 rows 71 us (3.7 TB/s); 700 rows, SwiGLU 1.36 ms (35 TFLOP/s). One form with 4 x 4 outputs a thread and
// element-wise loads, before: 647, 585 us and 2.15 ms. The tile form's limit is shared memory: 128 bytes a clock feed 8 x 8
// outputs a thread just at the multiply-adds' rate. 16-bit operands through registers, 2,048 rows, 4,096 x 4,090: 2.02 ms.
//
// Epilogues: store (optional bias), add into the 32-bit residual stream, or
// SwiGLU over a stacked [gate; up] weight (rows 0..N-1 gate, N..2N-1 up).
#include "common.cuh"

#define EPI_STORE 0
#define EPI_RESIDUAL 1
#define EPI_SWIGLU 2

int cuca_device_sms();

namespace {

constexpr int CHUNK = 64;  // products of one run
constexpr int FEW = 16;    // tokens of one block of the few-row form at most

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = ok ? 16 : 0;  // 0: nothing is read and the 16 bytes become zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two neighbouring elements from `src` on, of which `left` exist (zeros behind), and their values as floats; even: `src` is
// aligned to two elements.
__device__ __forceinline__ float2 load_two(const float* src, int left, bool even) {
  if (even && left >= 2) return *reinterpret_cast<const float2*>(src);
  return make_float2(left >= 1 ? src[0] : 0.f, left >= 2 ? src[1] : 0.f);
}
__device__ __forceinline__ uint32_t load_two(const __nv_bfloat16* src, int left, bool even) {
  if (even && left >= 2) return *reinterpret_cast<const uint32_t*>(src);
  const uint16_t* u = reinterpret_cast<const uint16_t*>(src);
  return (left >= 1 ? u[0] : 0u) | (left >= 2 ? (uint32_t)u[1] << 16 : 0u);
}
__device__ __forceinline__ float2 to_f32x2(float2 t) { return t; }
__device__ __forceinline__ float2 to_f32x2(uint32_t t) { return make_float2(__uint_as_float(t << 16), __uint_as_float(t & 0xffff0000u)); }

// `v` (and for SwiGLU `u`): the sums of output (m, n)
template <typename TI, typename TO, int EPI>
__device__ __forceinline__ void finish(TO* out, const TI* bias, size_t o, int n, float v, float u) {
  if (EPI == EPI_SWIGLU) {
    out[o] = from_f32<TO>(v / (1.f + expf(-v)) * u);
  } else {
    if (bias) v += to_f32(bias[n]);
    if (EPI == EPI_RESIDUAL) out[o] = from_f32<TO>(to_f32(out[o]) + v);
    else out[o] = from_f32<TO>(v);
  }
}

// ---- few rows
// A block: NB weight rows (SwiGLU: NB / 2 gate rows and their up rows) x MT tokens x all of K, in rounds of RC runs.
// Thread (n, c) sums run c of row n for the MT tokens; then thread (n, m) adds the round's RC sums in order. Runs lie
// PITCH floats apart in shared memory: a warp's 16-byte reads of 32 runs meet no bank conflict, and the tokens' values
// are read by 16 lanes at once.
template <int MT>
struct Rows {
  static constexpr int NB = 16;
  static constexpr int RC = MT <= 4 ? 16 : 8;
  static constexpr int THREADS = NB * RC;
  static constexpr int STAGES = MT == 8 ? 3 : 2;
  static constexpr int PITCH = CHUNK + 4;
  static constexpr int STAGE = (NB + MT) * RC * PITCH;  // floats
  static constexpr int SMEM = (STAGES * STAGE + RC * NB * MT + NB * MT) * 4;
  static constexpr int ITEMS = (NB * MT + THREADS - 1) / THREADS;
};

template <typename TI, typename TO, int MT, int EPI, bool VEC>
__global__ void __launch_bounds__(Rows<MT>::THREADS)
rows_kernel(const TI* __restrict__ A, const TI* __restrict__ W, const TI* __restrict__ bias, TO* __restrict__ out, int M,
            int N, int K, int lda, int ldo) {
  using C = Rows<MT>;
  constexpr bool DUAL = EPI == EPI_SWIGLU;
  constexpr int NB = C::NB, RC = C::RC, P = C::PITCH, RK = RC * CHUNK;  // RK: K of one round
  constexpr int OUTS = DUAL ? NB / 2 : NB;                              // outputs of a block
  extern __shared__ __align__(16) float sm[];
  float* part = sm + C::STAGES * C::STAGE;  // [RC][NB][MT]
  float* sums = part + RC * NB * MT;        // [NB][MT], SwiGLU only: gate beside up
  const int n0 = blockIdx.x * OUTS, m0 = blockIdx.y * MT;
  const int rounds = (K + RK - 1) / RK;
  auto row_of = [&](int r) { return !DUAL ? n0 + r : (r < OUTS ? n0 + r : N + n0 + r - OUTS); };
  auto row_ok = [&](int r) { return (DUAL ? n0 + r % OUTS : n0 + r) < N; };
  // rows of `src` (row r, K run) into runs [RC][rows][P]
  auto load_w = [&](int round, float* dst) {
    if (VEC) {
      for (int e = threadIdx.x; e < NB * RK / 4; e += C::THREADS) {
        const int r = e / (RK / 4), k = e % (RK / 4) * 4, gk = round * RK + k;
        const bool ok = row_ok(r) && gk < K;
        cp_async16(dst + ((k / CHUNK) * NB + r) * P + k % CHUNK, (const float*)W + (ok ? (size_t)row_of(r) * K + gk : 0), ok);
      }
    } else {
      for (int e = threadIdx.x; e < NB * RK; e += C::THREADS) {
        const int r = e / RK, k = e % RK, gk = round * RK + k;
        dst[((k / CHUNK) * NB + r) * P + k % CHUNK] = row_ok(r) && gk < K ? to_f32(W[(size_t)row_of(r) * K + gk]) : 0.f;
      }
    }
  };
  auto load_a = [&](int round, float* dst) {
    if (VEC) {
      for (int e = threadIdx.x; e < MT * RK / 4; e += C::THREADS) {
        const int r = e / (RK / 4), k = e % (RK / 4) * 4, gk = round * RK + k;
        const bool ok = m0 + r < M && gk < K;
        cp_async16(dst + ((k / CHUNK) * MT + r) * P + k % CHUNK, (const float*)A + (ok ? (size_t)(m0 + r) * lda + gk : 0), ok);
      }
    } else {
      for (int e = threadIdx.x; e < MT * RK; e += C::THREADS) {
        const int r = e / RK, k = e % RK, gk = round * RK + k;
        dst[((k / CHUNK) * MT + r) * P + k % CHUNK] = m0 + r < M && gk < K ? to_f32(A[(size_t)(m0 + r) * lda + gk]) : 0.f;
      }
    }
  };
  auto stage_w = [&](int round) { return sm + (round % C::STAGES) * C::STAGE; };
  auto stage_a = [&](int round) { return stage_w(round) + NB * RC * P; };
  pdl_trigger();
  if (VEC) {
    // the weights are no earlier kernel's output: the first rounds' are requested before the wait for the predecessor
    for (int s = 0; s < C::STAGES - 1 && s < rounds; ++s) load_w(s, stage_w(s));
    pdl_wait();
    for (int s = 0; s < C::STAGES - 1; ++s) {
      if (s < rounds) load_a(s, stage_a(s));
      cp_commit();
    }
  } else {
    pdl_wait();
  }
  const int n = threadIdx.x % NB, c = threadIdx.x / NB;
  float total[C::ITEMS];
#pragma unroll
  for (int i = 0; i < C::ITEMS; ++i) total[i] = 0.f;
  for (int round = 0; round < rounds; ++round) {
    if (VEC) {
      const int next = round + C::STAGES - 1;  // into the stage that the round before this one has left
      if (next < rounds) {
        load_w(next, stage_w(next));
        load_a(next, stage_a(next));
      }
      cp_commit();
      cp_wait<C::STAGES - 1>();
    } else {
      load_w(round, stage_w(round));
      load_a(round, stage_a(round));
    }
    __syncthreads();
    float acc[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = 0.f;
    const float4* w4 = reinterpret_cast<const float4*>(stage_w(round) + (c * NB + n) * P);
    const float* at = stage_a(round) + c * MT * P;
#pragma unroll 4
    for (int q = 0; q < CHUNK / 4; ++q) {
      const float4 w = w4[q];
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const float4 a = *reinterpret_cast<const float4*>(at + m * P + 4 * q);
        acc[m] = fmaf(a.x, w.x, acc[m]);
        acc[m] = fmaf(a.y, w.y, acc[m]);
        acc[m] = fmaf(a.z, w.z, acc[m]);
        acc[m] = fmaf(a.w, w.w, acc[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) part[(c * NB + n) * MT + m] = acc[m];
    __syncthreads();
    const int runs = min(RC, (K - round * RK + CHUNK - 1) / CHUNK);
#pragma unroll
    for (int i = 0; i < C::ITEMS; ++i) {
      const int e = threadIdx.x + i * C::THREADS;
      if (e < NB * MT)
        for (int r = 0; r < runs; ++r) total[i] += part[r * NB * MT + e];
    }
    __syncthreads();  // the stage and the sums are free again
  }
#pragma unroll
  for (int i = 0; i < C::ITEMS; ++i) {
    const int e = threadIdx.x + i * C::THREADS;
    if (e >= NB * MT) continue;
    if (DUAL) {
      sums[e] = total[i];
    } else {
      const int gn = n0 + e / MT, gm = m0 + e % MT;
      if (gn < N && gm < M) finish<TI, TO, EPI>(out, bias, (size_t)gm * ldo + gn, gn, total[i], 0.f);
    }
  }
  if (DUAL) {
    __syncthreads();
    for (int e = threadIdx.x; e < OUTS * MT; e += C::THREADS) {
      const int gn = n0 + e / MT, gm = m0 + e % MT;
      if (gn < N && gm < M)
        finish<TI, TO, EPI>(out, bias, (size_t)gm * ldo + gn, gn, sums[e], sums[e + OUTS * MT]);
    }
  }
}

// ---- many rows
// A block: BM tokens x BN weight rows (SwiGLU: BN / 2 gate rows and their up rows), K in steps of BK. Operands stay
// K-major in shared memory, PITCH floats a row, and a thread reads four K at a time of its rows (BM / TM apart) and
// columns (BN / 8 apart): neighbouring lanes read neighbouring rows, which PITCH spreads over all banks.
template <int BM, int BN, int TM, bool VEC>
struct Tile {
  static constexpr int BK = 32, PITCH = BK + 4, TN = 8;
  static constexpr int RT = BM / TM, CT = BN / TN;  // threads along rows, columns
  static constexpr int THREADS = RT * CT;
  static constexpr int STAGES = 3;
  static constexpr int STAGE = (BM + BN) * PITCH;  // floats
  static constexpr int SMEM = STAGES * STAGE * 4;
  static constexpr int BLOCKS = BM == 128 ? 1 : VEC ? 3 : 2;  // a SM
};

template <typename TI, typename TO, int BM, int BN, int TM, int EPI, bool VEC>
__global__ void __launch_bounds__((Tile<BM, BN, TM, VEC>::THREADS), (Tile<BM, BN, TM, VEC>::BLOCKS))
tile_kernel(const TI* __restrict__ A, const TI* __restrict__ W, const TI* __restrict__ bias, TO* __restrict__ out, int M,
            int N, int K, int lda, int ldo) {
  using C = Tile<BM, BN, TM, VEC>;
  constexpr bool DUAL = EPI == EPI_SWIGLU;
  constexpr int TN = C::TN, P = C::PITCH, BK = C::BK, OUTS = DUAL ? BN / 2 : BN;
  extern __shared__ __align__(16) float sm[];
  const int tiles_m = (M + BM - 1) / BM;  // neighbouring blocks share weight rows
  const int n0 = blockIdx.x / tiles_m * OUTS, m0 = blockIdx.x % tiles_m * BM;
  const int tx = threadIdx.x % C::CT, ty = threadIdx.x / C::CT;
  const int steps = (K + BK - 1) / BK;
  auto row_of = [&](int r) { return !DUAL ? n0 + r : (r < OUTS ? n0 + r : N + n0 + r - OUTS); };
  auto row_ok = [&](int r) { return (DUAL ? n0 + r % OUTS : n0 + r) < N; };
  auto load = [&](int step) {
    float* dst = sm + (step % C::STAGES) * C::STAGE;
#pragma unroll
    for (int e = threadIdx.x; e < (BM + BN) * BK / 4; e += C::THREADS) {
      const int r = e / (BK / 4), k = e % (BK / 4) * 4, gk = step * BK + k;
      const bool is_a = r < BM;
      const bool ok = (is_a ? m0 + r < M : row_ok(r - BM)) && gk < K;
      const float* src = is_a ? (const float*)A + (ok ? (size_t)(m0 + r) * lda + gk : 0)
                              : (const float*)W + (ok ? (size_t)row_of(r - BM) * K + gk : 0);
      cp_async16(dst + r * P + k, src, ok);
    }
  };
  // through registers: the elements of a step are requested a step before they are put down
  constexpr int TWOS = VEC ? 1 : (BM + BN) * BK / 2 / C::THREADS;
  const bool even = !VEC && ((K | lda) & 1) == 0 && (((uintptr_t)A | (uintptr_t)W) & (2 * sizeof(TI) - 1)) == 0;
  decltype(load_two(A, 0, false)) held[TWOS];
  auto fetch = [&](int step) {
#pragma unroll
    for (int i = 0; i < TWOS; ++i) {
      const int e = threadIdx.x + i * C::THREADS, r = e / (BK / 2), gk = step * BK + e % (BK / 2) * 2;
      const bool is_a = r < BM, ok = is_a ? m0 + r < M : row_ok(r - BM);
      held[i] = load_two(is_a ? A + (size_t)(m0 + r) * lda + gk : W + (size_t)row_of(r - BM) * K + gk, ok ? K - gk : 0, even);
    }
  };
  auto put = [&](int step) {
#pragma unroll
    for (int i = 0; i < TWOS; ++i) {
      const int e = threadIdx.x + i * C::THREADS;
      *reinterpret_cast<float2*>(sm + (step % C::STAGES) * C::STAGE + e / (BK / 2) * P + e % (BK / 2) * 2) = to_f32x2(held[i]);
    }
  };
  pdl_trigger();
  pdl_wait();
  float acc[TM][TN], total[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = total[i][j] = 0.f;
  if constexpr (VEC) {
    for (int s = 0; s < C::STAGES - 1; ++s) {
      if (s < steps) load(s);
      cp_commit();
    }
  } else {
    fetch(0);
    put(0);
    if (steps > 1) fetch(1);
  }
  for (int step = 0; step < steps; ++step) {
    if constexpr (VEC) cp_wait<C::STAGES - 2>();
    __syncthreads();  // this step's tiles have landed, and the stage of the step before is free
    if constexpr (VEC) {
      if (step + C::STAGES - 1 < steps) load(step + C::STAGES - 1);
      cp_commit();
    } else {
      if (step + 1 < steps) put(step + 1);
      if (step + 2 < steps) fetch(step + 2);
    }
    const float* as = sm + (step % C::STAGES) * C::STAGE;
    const float* at = as + ty * P;
    const float* bt = as + (BM + tx) * P;
#pragma unroll
    for (int q = 0; q < BK / 4; ++q) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(at + i * C::RT * P + 4 * q);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 b = *reinterpret_cast<const float4*>(bt + j * C::CT * P + 4 * q);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
      }
    }
    if ((step + 1) % (CHUNK / BK) == 0 || step + 1 == steps) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          total[i][j] += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty + i * C::RT;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < (DUAL ? TN / 2 : TN); ++j) {
      const int gn = n0 + tx + j * C::CT;
      if (gn < N)
        finish<TI, TO, EPI>(out, bias, (size_t)gm * ldo + gn, gn, total[i][j], total[i][DUAL ? j + TN / 2 : j]);
    }
  }
}

template <typename TI, typename TO, int MT, int EPI, bool VEC>
int launch_rows(const void* A, const void* W, const void* bias, void* out, int M, int N, int K, int lda, int ldo,
                cudaStream_t stream) {
  using C = Rows<MT>;
  constexpr int OUTS = EPI == EPI_SWIGLU ? C::NB / 2 : C::NB;
  auto kernel = rows_kernel<TI, TO, MT, EPI, VEC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  CUCA_REQUIRE(e == cudaSuccess, "gemm: %d bytes of shared memory were refused: %s", C::SMEM, cudaGetErrorString(e));
  cuca_launch(kernel, dim3((N + OUTS - 1) / OUTS, (M + MT - 1) / MT), dim3(C::THREADS), C::SMEM, stream, true, (const TI*)A,
              (const TI*)W, (const TI*)bias, (TO*)out, M, N, K, lda, ldo);
  return 0;
}

template <typename TI, typename TO, int BM, int BN, int TM, int EPI, bool VEC>
int launch_tile(const void* A, const void* W, const void* bias, void* out, int M, int N, int K, int lda, int ldo,
                cudaStream_t stream) {
  using C = Tile<BM, BN, TM, VEC>;
  constexpr int OUTS = EPI == EPI_SWIGLU ? BN / 2 : BN;
  auto kernel = tile_kernel<TI, TO, BM, BN, TM, EPI, VEC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  CUCA_REQUIRE(e == cudaSuccess, "gemm: %d bytes of shared memory were refused: %s", C::SMEM, cudaGetErrorString(e));
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + OUTS - 1) / OUTS);
  CUCA_REQUIRE(tiles < (1ll << 31), "gemm: %d x %d outputs are too many", M, N);
  cuca_launch(kernel, dim3((unsigned)tiles), dim3(C::THREADS), C::SMEM, stream, true, (const TI*)A, (const TI*)W,
              (const TI*)bias, (TO*)out, M, N, K, lda, ldo);
  return 0;
}

template <typename TI, typename TO, int EPI, bool VEC>
int launch_form(const void* A, const void* W, const void* bias, void* out, int M, int N, int K, int lda, int ldo,
                cudaStream_t stream) {
  constexpr int OUTS64 = EPI == EPI_SWIGLU ? 32 : 64;
#define ROWS(MT) return launch_rows<TI, TO, MT, EPI, VEC>(A, W, bias, out, M, N, K, lda, ldo, stream)
#define TILE(BM, BN, TM) return launch_tile<TI, TO, BM, BN, TM, EPI, VEC>(A, W, bias, out, M, N, K, lda, ldo, stream)
  const long long blocks_64 = (long long)((M + 63) / 64) * ((N + OUTS64 - 1) / OUTS64);
  const long long blocks_128 = (long long)((M + 127) / 128) * ((N + 2 * OUTS64 - 1) / (2 * OUTS64));
  if (M <= 1) ROWS(1);
  if (M <= 2) ROWS(2);
  if (M <= 4) ROWS(4);
  if (M <= 8) ROWS(8);
  // Above 16 rows the few-row form reads the weights again for every 16 (from L2), and the tile form leaves SMs idle
  // unless there are many tiles. Measured on K = 2048, us (few-row, tiles of 64): N = 2048, 64 rows 73, 98; 96 rows
  // 104, 98; N = 3072, 48 rows 66, 86; 64 rows 94, 86; N = 32000, 24 rows 418, 270
  if (M <= FEW || (M <= 64 && blocks_64 * ((M + 15) / 16) < 160)) ROWS(16);
  // A SM works through a tile of 128 alone in the time of 3.3 tiles of 64 (three at once): the larger one is 10 %
  // faster where its last round is full. Measured on K = 2048, us (64, 128): N = 3072, 700 rows 272, 234; N = 2048,
  // 700 rows 211, 258; SwiGLU N = 8192, 128 rows 279, 236; 1400 rows 2481, 2250
  const long long sms = cuca_device_sms(), rounds_64 = (blocks_64 + sms - 1) / sms, rounds_128 = (blocks_128 + sms - 1) / sms;
  if (10 * rounds_128 <= 3 * rounds_64) TILE(128, 128, 8);
  TILE(64, 64, 4);
#undef ROWS
#undef TILE
}

template <typename TI, typename TO, int EPI>
int launch(const void* A, const void* W, const void* bias, void* out, int M, int N, int K, int lda, int ldo,
           cudaStream_t stream) {
  const bool vec = sizeof(TI) == 4 && K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  if (sizeof(TI) == 4 && vec) return launch_form<TI, TO, EPI, sizeof(TI) == 4>(A, W, bias, out, M, N, K, lda, ldo, stream);
  return launch_form<TI, TO, EPI, false>(A, W, bias, out, M, N, K, lda, ldo, stream);
}

}  // namespace

// out = epilogue(A[M,K] W[N,K]^T). in_dtype: A, W and bias; out_dtype: out.
// epilogue 0 store, 1 out (32-bit) += result, 2 SwiGLU (W has 2N rows).
CUCA_API int cuca_gemm_simt(const void* A, const void* W, const void* bias, void* out, int in_dtype, int out_dtype,
                   int M, int N, int K, int lda, int ldo, int epilogue, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  CUCA_REQUIRE(K > 0 && lda >= K && ldo >= N, "gemm: bad sizes M=%d N=%d K=%d lda=%d ldo=%d", M, N, K, lda, ldo);
  CUCA_REQUIRE(epilogue != EPI_RESIDUAL || out_dtype == CUCA_F32, "gemm: the residual stream is 32-bit");
  CUCA_REQUIRE(epilogue != EPI_SWIGLU || bias == nullptr, "gemm: SwiGLU takes no bias");
  int rc = 0;
#define GO(TI, TO)                                                                                                 \
  do {                                                                                                             \
    if (epilogue == EPI_STORE) rc = launch<TI, TO, EPI_STORE>(A, W, bias, out, M, N, K, lda, ldo, stream);          \
    else if (epilogue == EPI_RESIDUAL) rc = launch<TI, float, EPI_RESIDUAL>(A, W, bias, out, M, N, K, lda, ldo, stream); \
    else if (epilogue == EPI_SWIGLU) rc = launch<TI, TO, EPI_SWIGLU>(A, W, bias, out, M, N, K, lda, ldo, stream);   \
    else CUCA_REQUIRE(false, "gemm: unknown epilogue %d", epilogue);                                                \
  } while (0)
  if (in_dtype == CUCA_F32 && out_dtype == CUCA_F32) GO(float, float);
  else if (in_dtype == CUCA_BF16 && out_dtype == CUCA_BF16) GO(__nv_bfloat16, __nv_bfloat16);
  else if (in_dtype == CUCA_BF16 && out_dtype == CUCA_F32) GO(__nv_bfloat16, float);
  else CUCA_REQUIRE(false, "gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
#undef GO
  if (rc) return rc;
  CUCA_CHECK_LAUNCH("gemm_simt");
  return 0;
}
