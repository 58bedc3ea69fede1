// 32-bit contraction out = A[M,K] * W[N,K]^T on the 5th-generation tensor cores: the true 32-bit path of every projection,
// and the bfloat16 path's stand-in for shapes that its own kernel refuses.
//
// A 32-bit value from 2^-110 on is the sum of three bfloat16 parts, exactly: the nearest bfloat16 number, the nearest to what
// is left, and the rest, at most 2^-8 and 2^-16 of the value's power of two. Of the nine products of two values' parts the six
// largest count; the others come to at most 2^-23 of the product, 2^-28 on average, of either sign. tcgen05.mma sums
// them in 32 bits, and the tensor cores cut off where a 32-bit addition rounds. So the largest products, which take 16 bits
// each, have an accumulator of their own over a chunk of 64 products, where little is left to cut off, and the five others,
// a 2^-8th as large, one over a block of four chunks. Everything else is added with rounding: the chunks' sums of a block and its small
// products, and the blocks' in ascending order. What 32 bits hold exactly (whole numbers, one product with a power of
// two) comes out exactly. Each output is summed in this one order whatever M and the kernel's form are, so a row's result never depends
// on the rest of the batch. A warp computes an output again with plain multiply-adds where the total is no finite number (an infinite
// value has no parts) or a tiny one, and where values below 2^-110 that lost something in their parts (the converters note whose
// rows have any) may matter beside it: see `settled`.
// Error against 64 bits, relative 2-norm, normal values (multiply-adds in runs of 64 in brackets): K = 1 2.6e-8 (2.5e-8), 16
// 3.5e-8 (7.3e-8), 2,048 9.8e-8 (1.8e-7), 8,192 1.3e-7 (2.5e-7); values of one sign, where what is cut off adds up, K = 64
// 9.0e-8 (1.2e-7), 256 9.1e-8 (7.3e-8), 2,048 9.3e-8 (9.2e-8), 8,192 1.2e-7 (1.8e-7). With one accumulator for all products and a unit in the last place given
// back to every chunk for what is cut off, sums that are exact came out wrong (1 x 1) and K = 1 had 6.5e-8.
//
// The weights are the 128-row operand, the tokens the columns. A CTA (one an SM): the copy engine streams weight chunks
// into a ring as they are; converter warps split them, a row a lane, into tensor memory, from where the tensor cores read
// them (shared memory would not stand their 24 reads of a part); the tokens' parts lie in shared memory, converted by two
// warps over few tokens, or by a kernel of its own before (`split_kernel`) from 17 tokens on, since every block of weight rows
// reads them; eight or four warps add the chunks' sums up. Few tiles: a cluster of up to eight CTAs shares a tile's K, each
// keeps its blocks' sums, and all add them in order out of each other's shared memory. Operands that take no copies
// (16-bit ones, K or a row stride not a multiple of 4, an address off 16 bytes) come element by element with the same results:
// 4,096 x 4,090, us, multiply-adds and this: 2,048 tokens 32-bit 2,398, 650, 16-bit 2,018, 960; 16 tokens 244, 37 and 240, 38.
//
// Epilogues: store (optional bias), add into the 32-bit residual stream, or SwiGLU over a stacked [gate; up] weight (rows
// 0..N-1 gate, N..2N-1 up).
#include "tcgen05.cuh"
#include "f32x2.cuh"
#include <algorithm>
#include <type_traits>

#define EPI_STORE 0
#define EPI_RESIDUAL 1
#define EPI_SWIGLU 2

namespace {

constexpr int CHUNK = TILE_K;         // products that one accumulator sums: 64
constexpr int BLOCK = 4;              // chunks whose sums are added up before they meet the total
constexpr int ROWS = TILE_A;          // weight rows of a tile
constexpr int ROW_BYTES = CHUNK * 2;  // one row of one part in shared memory: one swizzle span
constexpr int MAX_CLUSTER = 8;
constexpr int PRE_TOKENS = 32;        // tiles of so many tokens and more take the tokens' parts from memory
constexpr int FEW_TOKENS = 16;        // up to here 16-byte copies of the weights start before the kernel ahead is done
constexpr int SPLIT_RUN = 2048;       // elements of a row that one block of `split_kernel` takes

template <typename TI> struct Parts { static constexpr int N = 3; };
template <> struct Parts<__nv_bfloat16> { static constexpr int N = 1; };  // (the others would be zeros)

struct GemmParams {
  const void* A;
  const void* W;
  const void* bias;
  void* out;
  int* err;
  int M, N, K, lda, ldo;
  int epilogue, out_f32;
  const uint16_t* marks;  // of the tokens, [M][runs of SPLIT_RUN], where their parts come from memory
  int tiles_m;  // token tiles
  int slices;   // CTAs of a cluster that share a tile's K
};

struct Marks;
struct MarksByTwo;

template <typename TI, int NT>
struct Form {
  static constexpr int P = Parts<TI>::N;
  static constexpr bool PRE = NT >= PRE_TOKENS;  // the tokens' parts come from memory, else from converters of this kernel
  using RowMarks = std::conditional_t<PRE, Marks, MarksByTwo>;
  // warps: sums, weight converters (eight a set; two sets take chunks in turn), the tokens' (converters, or one that copies),
  // the ring's loader, contractions
  static constexpr int EPI_WARPS = PRE ? 8 : 4;
  static constexpr int SETS = PRE ? 1 : 2;
  static constexpr int A_WARPS = 8 * SETS;
  static constexpr int B_WARPS = PRE ? 1 : 2;
  static constexpr int A_WARP = EPI_WARPS, B_WARP = A_WARP + A_WARPS, LOAD_WARP = B_WARP + B_WARPS, MMA_WARP = LOAD_WARP + 1;
  static constexpr int THREADS = 32 * (MMA_WARP + 1);
  static constexpr int COLS = NT / (EPI_WARPS / 4);  // tokens of one summing thread
  // weights as they are: a ring of chunks, filled by the copy engine
  static constexpr int RAW = ROWS * CHUNK * 4;
  static constexpr int RAWS = NT > 64 ? 3 : PRE ? 4 : 6;
  // a chunk of the parts: the weights' in tensor memory, the tokens' in shared memory
  static constexpr int STAGES = PRE ? 2 : 3;
  static constexpr int A_COLS = P * CHUNK / 2;
  static constexpr int B_BYTES = P * NT * ROW_BYTES;
  static constexpr int PASS_ROWS = B_WARPS * 2;  // 16 threads a token row, 16 bytes each
  static constexpr int PASSES = NT / PASS_ROWS;
  // columns of tensor memory: two accumulators of the largest products, one of the small ones, the parts, then the total (with
  // slices: the sums of this CTA's blocks but for the last, which stays in registers), which lies in shared memory where
  // there is no room left
  static constexpr int SMALL_AT = 2 * NT, A_AT = (P == 3 ? 3 : 2) * NT, SUM_AT = A_AT + STAGES * A_COLS;
  static constexpr bool SUM_IN_SMEM = SUM_AT + NT > 512;
  static constexpr int DATA = RAWS * RAW + STAGES * B_BYTES;
  static constexpr int SUM_BYTES = SUM_IN_SMEM ? NT * ROWS * 4 : 0;
  static constexpr int SMEM = DATA + SUM_BYTES + 1024 + 256 + (ROWS + NT + 4) * 4;
  static constexpr int BLOCKS_HELD = SUM_IN_SMEM ? 0 : std::min((512 - SUM_AT) / NT + 1, DATA / (NT * ROWS * 4));
  static_assert(SUM_AT <= 512 && SMEM <= 227 * 1024, "tensor or shared memory");
};

__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
  const int n = valid ? 4 : 0;  // 0: nothing is read and the 4 bytes become zeros
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t local, uint32_t rank, uint32_t offset) {
  uint32_t a, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a + offset) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster(uint32_t local, uint32_t rank, uint32_t offset) {
  return __uint_as_float(ld_cluster_u32(local, rank, offset));
}

// What is noted of a row (of weights or of a token): a value whose three parts are not all of it (one below 2^-110, whose lower
// bits bfloat16 does not hold; up to 2^-133 of it is lost), one of at least 2^40.
constexpr uint32_t LOSSY = 1, LARGE = 2;
struct Marks {
  uint32_t lost = 0;  // the third parts' bits, of which bfloat16 holds the upper half
  float most = 0.f;
  __device__ __forceinline__ void see(float4 v, uint2) {
    most = fmaxf(most, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
  }
  __device__ __forceinline__ uint32_t word() const { return (lost << 16 ? LOSSY : 0) | (most >= 1.09951163e12f ? LARGE : 0); }
};
// The same, the largest of the first parts, two a step: where the converters set the pace (tiles of 16 tokens: 2,048 x 8,192, a CTA a
// tile, 86 -> 83 us; in tiles of 96, which have no registers for it, 320 -> 326).
struct MarksByTwo {
  uint32_t lost = 0;
  __nv_bfloat162 most = __floats2bfloat162_rn(0.f, 0.f);
  __device__ __forceinline__ void see(float4, uint2 part) {
    most = __hmax2(most, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&part.x)));
    most = __hmax2(most, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&part.y)));
  }
  __device__ __forceinline__ uint32_t word() const {
    return (lost << 16 ? LOSSY : 0) | (__bfloat162float(__hmax(most.x, most.y)) >= 1.09951163e12f ? LARGE : 0);
  }
};
// Whether a total stands. Finite, and not so small (2^-100) that products of small parts may have been lost; and where a row lost
// something of its values, they met none of 2^40 or more and the total is no less than 2^-50, beside which K times 2^-93 is nothing.
__device__ __forceinline__ bool settled(float v, uint32_t token, uint32_t weight) {
  const float a = fabsf(v);
  if (!(a <= 3.402823466e38f && (a >= 7.888609e-31f || a == 0.f))) return false;
  if (!((token | weight) & LOSSY)) return true;
  return a >= 8.8817842e-16f && !((token & LOSSY) && (weight & LARGE)) && !((weight & LOSSY) && (token & LARGE));
}
// One output by a warp with plain multiply-adds.
template <typename TI>
__device__ float dot_again(const TI* a, const TI* w, int K) {
  const int lane = threadIdx.x & 31;
  float s = 0.f;
  for (int k0 = 0; k0 < K; k0 += 128) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + 32 * j + lane;
      if (k < K) s = fmaf(to_f32(a[k]), to_f32(w[k]), s);
    }
    if (__any_sync(0xffffffffu, isnan(s))) return __int_as_float(0x7fc00000);
  }
  return warp_sum(s);
}
// `v` of this lane's output (token m, weight row w), computed again where `again`; the whole warp comes here.
template <typename TI>
__device__ __noinline__ float settle(const GemmParams& p, float v, bool again, int m, int w) {
  unsigned todo = __ballot_sync(0xffffffffu, again);
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const int mm = __shfl_sync(0xffffffffu, m, src), ww = __shfl_sync(0xffffffffu, w, src);
    const float r = dot_again((const TI*)p.A + (size_t)mm * p.lda, (const TI*)p.W + (size_t)ww * p.K, p.K);
    if ((int)(threadIdx.x & 31) == src) v = r;
  }
  return v;
}

// `v` (and for SwiGLU `u`): the sums of output (m, n)
template <typename TI>
__device__ __forceinline__ void finish(const GemmParams& p, int m, int n, float v, float u) {
  const size_t o = (size_t)m * p.ldo + n;
  if (p.epilogue == EPI_SWIGLU) v = v / (1.f + expf(-v)) * u;
  else if (p.bias) v += to_f32(((const TI*)p.bias)[n]);
  if (p.out_f32) {
    float* out = (float*)p.out + o;
    *out = p.epilogue == EPI_RESIDUAL ? *out + v : v;
  } else {
    ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(v);
  }
}

// Four neighbouring elements from `src` on: of a row of which `left` elements are there (VEC: all four).
template <bool VEC>
__device__ __forceinline__ float4 load4(const float* src, int left) {
  if (VEC) return __ldg(reinterpret_cast<const float4*>(src));
  return make_float4(left > 0 ? __ldg(src) : 0.f, left > 1 ? __ldg(src + 1) : 0.f, left > 2 ? __ldg(src + 2) : 0.f,
                     left > 3 ? __ldg(src + 3) : 0.f);
}
template <bool VEC>
__device__ __forceinline__ uint2 load4(const __nv_bfloat16* src, int left) {
  const uint16_t* u = reinterpret_cast<const uint16_t*>(src);
  const uint32_t a = left > 0 ? __ldg(u) : 0, b = left > 1 ? __ldg(u + 1) : 0, c = left > 2 ? __ldg(u + 2) : 0,
                 d = left > 3 ? __ldg(u + 3) : 0;
  return make_uint2(a | b << 16, c | d << 16);
}

// The bfloat16 numbers nearest to a and to b; a and b become what is left, exactly.
__device__ __forceinline__ uint32_t take_part(float& a, float& b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  const uint32_t part = *reinterpret_cast<const uint32_t*>(&t);
  const f32x2 up = f2_pack(__uint_as_float(part << 16), __uint_as_float(part & 0xffff0000u));
  f2_unpack(f2_fma(up, f2_both(-1.f), f2_pack(a, b)), a, b);
  return part;
}
__device__ __forceinline__ uint32_t upper_halves(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
// four elements' parts
template <typename M>
__device__ __forceinline__ void split(uint2 (&w)[3], float4 v, M& marks) {
  const float4 whole = v;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    w[t].x = take_part(v.x, v.y);
    w[t].y = take_part(v.z, v.w);
  }
  marks.see(whole, w[0]);
  marks.lost |= __float_as_uint(v.x) | __float_as_uint(v.y) | __float_as_uint(v.z) | __float_as_uint(v.w);
  w[2] = make_uint2(upper_halves(v.x, v.y), upper_halves(v.z, v.w));
}
template <typename M>
__device__ __forceinline__ void split(uint2 (&w)[1], uint2 v, M&) { w[0] = v; }
__device__ __forceinline__ void clear(float4& v) { v = make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ void clear(uint2& v) { v = make_uint2(0, 0); }

// The tokens' parts, [part][token][ld] in bf16, and their marks: a block takes SPLIT_RUN elements of a row. Bound by its bytes.
template <typename TI, bool VEC>
__global__ void __launch_bounds__(256)
split_kernel(const TI* __restrict__ A, __nv_bfloat16* __restrict__ parts, uint16_t* __restrict__ out_marks, int m0, int M, int K, int lda, int ld) {
  constexpr int P = Parts<TI>::N, QUADS = SPLIT_RUN / 4 / 256;
  pdl_trigger();
  pdl_wait();
  const int m = m0 + blockIdx.y, k0 = blockIdx.x * SPLIT_RUN + threadIdx.x * 4;
  decltype(load4<VEC>(A, 0)) v[QUADS];
#pragma unroll
  for (int i = 0; i < QUADS; ++i) {
    const int k = k0 + i * 1024;
    if (k < K) v[i] = load4<VEC>(A + (size_t)m * lda + k, K - k);
    else clear(v[i]);
  }
  Marks marks;
#pragma unroll
  for (int i = 0; i < QUADS; ++i) {
    const int k = k0 + i * 1024;
    uint2 w[P];
    split(w, v[i], marks);
    if (k < K)
#pragma unroll
      for (int t = 0; t < P; ++t) *reinterpret_cast<uint2*>(parts + ((size_t)t * M + m) * ld + k) = w[t];
  }
  if (P == 3) {
    const uint32_t word = marks.word();
    const int lossy = __syncthreads_or(word & LOSSY), large = __syncthreads_or(word & LARGE);
    if (threadIdx.x == 0) out_marks[(size_t)m * gridDim.x + blockIdx.x] = (lossy ? LOSSY : 0) | (large ? LARGE : 0);
  }
}

template <typename TI, int NT, bool VEC>
__global__ void __launch_bounds__((Form<TI, NT>::THREADS), 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const GemmParams p) {
  using C = Form<TI, NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* tokens = smem + C::RAWS * C::RAW;
  float* total_s = (float*)(smem + C::DATA);  // (with SUM_IN_SMEM: [token][row])
  uint64_t* raw_full = (uint64_t*)(smem + C::DATA + C::SUM_BYTES);
  uint64_t* raw_empty = raw_full + C::RAWS;
  uint64_t* full = raw_empty + C::RAWS;
  uint64_t* done = full + C::STAGES;  // a stage's contraction: its parts are free and its accumulator complete
  uint64_t* acc_empty = done + C::STAGES;
  uint64_t* small_full = acc_empty + 2;  // a block's small products are complete
  uint64_t* small_empty = small_full + 1;
  uint32_t* tmem_slot = (uint32_t*)(small_empty + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  // marks of what this CTA has split: its weight rows, the tile's tokens, whether any row is lossy
  uint32_t* row_marks = tmem_slot + 2;
  uint32_t* token_marks = row_marks + ROWS;
  uint32_t* any_lossy = token_marks + NT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool dual = p.epilogue == EPI_SWIGLU;
  const int OUTS = dual ? ROWS / 2 : ROWS;
  const int cta = blockIdx.x / p.slices, rank = blockIdx.x % p.slices;
  const int n0 = cta / p.tiles_m * OUTS, m0 = cta % p.tiles_m * NT;  // neighbouring CTAs share weight rows
  const int chunks = (p.K + CHUNK - 1) / CHUNK, blocks = (chunks + BLOCK - 1) / BLOCK;
  const int first = rank * blocks / p.slices * BLOCK, last = min((rank + 1) * blocks / p.slices * BLOCK, chunks);

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::RAWS; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], 8);
    }
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full[s], 8 + C::B_WARPS);  // (the copying warp's arrival brings the bytes it waits for)
      mbar_init(&done[s], 1);
    }
    for (int b = 0; b < 2; ++b) mbar_init(&acc_empty[b], C::EPI_WARPS);
    mbar_init(small_full, 1);
    mbar_init(small_empty, C::EPI_WARPS);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (C::P == 3)
    for (int e = threadIdx.x; e < ROWS + NT + 1; e += C::THREADS) row_marks[e] = 0;
  auto note = [&](uint32_t* at, uint32_t word) {
    if (word) atomicOr(at, word);
    if (word & LOSSY) *any_lossy = 1;
  };
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == C::LOAD_WARP) {
    // ---- weights into the ring. Over few tokens no predecessor is waited for: there the weights must not be its output. Beyond,
    // where a launch's time is not that of the weights' first copies, and in the form through registers, they may be.
    if (VEC && lane == 0) {
      if (p.M > FEW_TOKENS) pdl_wait();
      const uint64_t once = l2_evict_first();
      for (int c = first, i = 0; c < last; ++c, ++i) {
        const int s = i % C::RAWS;
        if (!mbar_wait(&raw_empty[s], ((i / C::RAWS) & 1) ^ 1, p.err, abort_flag)) break;
        mbar_expect_tx(&raw_full[s], C::RAW);
        uint8_t* dst = smem + s * C::RAW;
        // boxes of 32 elements x 64 rows; SwiGLU's tile: 64 gate rows, then their 64 up rows
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int row = b & 1 ? (dual ? p.N + n0 : n0 + 64) : n0, k = c * CHUNK + (b >> 1) * 32;
          if (p.tiles_m == 1) tma_load_2d_hint(dst + b * (C::RAW / 4), &tmW, &raw_full[s], k, row, once);
          else tma_load_2d(dst + b * (C::RAW / 4), &tmW, &raw_full[s], k, row);
        }
      }
    }
    __syncwarp();
  } else if (warp == C::MMA_WARP) {
    // ---- contractions (the whole warp walks the chunks, see elect_one)
    for (int c = first, i = 0; c < last; ++c, ++i) {
      const int st = i % C::STAGES, buf = i & 1;
      if (!warp_wait(&acc_empty[buf], ((i >> 1) & 1) ^ 1, p.err, abort_flag)) break;
      if (!warp_wait(&full[st], (i / C::STAGES) & 1, p.err, abort_flag)) break;
      // The converters' writes to the async proxy: the fence stands here, on the path from the writes through the barrier to
      // the contraction, and not in the converters, where it would wait for their loads in flight.
      fence_proxy_async();
      tc_fence_after();
      const uint32_t a = tmem + C::A_AT + st * C::A_COLS, sb = smem_u32(tokens + st * C::B_BYTES);
      // products of the weights' part pa and the tokens' part pb
      auto contract = [&](uint32_t acc, int pa, int pb, bool add) {
        const uint32_t at = a + pa * CHUNK / 2;
        const uint64_t bd = smem_desc(sb + pb * NT * ROW_BYTES);
#pragma unroll
        for (int k = 0; k < CHUNK / UMMA_K; ++k)
          umma_bf16_tmem_a(acc, at + k * UMMA_K / 2, bd + k * UMMA_K * 2 / 16, instr_desc(NT), add || k > 0);
      };
      // The small products' one accumulator is drained while largest products are contracted: those of a block's last chunk
      // come behind its small ones, those of its first chunk before them.
      const bool begins = i % BLOCK == 0, ends = i % BLOCK == BLOCK - 1 || c == last - 1, ahead = C::P == 3 && begins && !ends;
      if (ahead && elect_one()) contract(tmem + buf * NT, 0, 0, false);
      __syncwarp();
      if (C::P == 3 && begins && !warp_wait(small_empty, ((i / BLOCK) & 1) ^ 1, p.err, abort_flag)) break;
      if (elect_one()) {
        if (C::P == 3) {  // the smallest first
          contract(tmem + C::SMALL_AT, 2, 0, !begins);
          contract(tmem + C::SMALL_AT, 0, 2, true);
          contract(tmem + C::SMALL_AT, 1, 1, true);
          contract(tmem + C::SMALL_AT, 1, 0, true);
          contract(tmem + C::SMALL_AT, 0, 1, true);
          if (ends) umma_commit(small_full);
        }
        if (!ahead) contract(tmem + buf * NT, 0, 0, false);
        umma_commit(&done[st]);
      }
      __syncwarp();
    }
  } else if (warp >= C::B_WARP) {
    pdl_wait();
    if constexpr (C::PRE) {
      // ---- the tokens' parts, one box of NT rows each. Rows past the end are the next part's or zeros: what they give is
      // never stored
      if (lane == 0) {
        for (int c = first, n = 0; c < last; ++c, ++n) {
          const int st = n % C::STAGES;
          if (!mbar_wait(&done[st], ((n / C::STAGES) & 1) ^ 1, p.err, abort_flag)) break;
          mbar_expect_tx(&full[st], C::B_BYTES);
#pragma unroll
          for (int t = 0; t < C::P; ++t)
            tma_load_2d(tokens + st * C::B_BYTES + t * NT * ROW_BYTES, &tmX, &full[st], c * CHUNK, t * p.M + m0);
        }
      }
      __syncwarp();
      if (C::P == 3) {
        const int runs = (p.K + SPLIT_RUN - 1) / SPLIT_RUN, items = min(NT, p.M - m0) * runs;
        for (int e = lane; e < items; e += 32) note(&token_marks[e / runs], p.marks[(size_t)m0 * runs + e]);
      }
    } else {
      // ---- the parts of the tokens: 16 threads a row, four elements each. Rows past the end are read from the last one
      const int pt = (warp - C::B_WARP) * 32 + lane, r0 = pt / 16, kq = pt % 16 * 4;
      const TI* rows[C::PASSES];
#pragma unroll
      for (int i = 0; i < C::PASSES; ++i) rows[i] = (const TI*)p.A + (size_t)min(m0 + r0 + i * C::PASS_ROWS, p.M - 1) * p.lda;
      decltype(load4<VEC>(rows[0], 0)) held[C::PASSES];
      // 16-byte loads stay inside their row; what they bring from before the end is cleared in the last chunk
      auto load = [&](int i, int c) {
        const int k = min(c, last - 1) * CHUNK + kq;
        return load4<VEC>(rows[i] + (VEC ? min(k, p.K - 4) : k), p.K - k);
      };
#pragma unroll
      for (int i = 0; i < C::PASSES; ++i) held[i] = load(i, first);
      const uint32_t at0 = r0 * ROW_BYTES + ((kq / 8 ^ (r0 & 7)) << 4) + (kq & 4) * 2;
      typename C::RowMarks marks[C::PASSES];
      for (int c = first, n = 0; c < last; ++c, ++n) {
        const int st = n % C::STAGES;
        if (VEC && (c + 1) * CHUNK > p.K && c * CHUNK + kq >= p.K) {
#pragma unroll
          for (int i = 0; i < C::PASSES; ++i) clear(held[i]);
        }
        uint2 parts[C::PASSES][C::P];
#pragma unroll
        for (int i = 0; i < C::PASSES; ++i) {
          split(parts[i], held[i], marks[i]);
          held[i] = load(i, c + 1);
        }
        if (!warp_wait(&done[st], ((n / C::STAGES) & 1) ^ 1, p.err, abort_flag)) break;
        uint8_t* sb = tokens + st * C::B_BYTES;
#pragma unroll
        for (int i = 0; i < C::PASSES; ++i)
#pragma unroll
          for (int t = 0; t < C::P; ++t)  // (a step of 4 rows modulo 8 turns bit 2 of the swizzled unit)
            *reinterpret_cast<uint2*>(sb + t * NT * ROW_BYTES + i * C::PASS_ROWS * ROW_BYTES + (at0 ^ (i * C::PASS_ROWS & 4) * 16)) = parts[i][t];
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[st]);
      }
      if (C::P == 3)
#pragma unroll
        for (int i = 0; i < C::PASSES; ++i) note(&token_marks[r0 + i * C::PASS_ROWS], marks[i].word());
    }
  } else if (warp >= C::A_WARP) {
    // ---- the parts of the weights: a row a lane, half of the chunk's K a warp
    const int cw = warp - C::A_WARP, quarter = warp & 3, half = (cw >> 2) & 1, set = cw >> 3;
    const int l = quarter * 32 + lane;
    const int raw_row = dual ? quarter * 16 + (lane & 15) + (lane & 16) * 4 : l;  // 16 gate rows and their 16 up rows take turns
    const uint32_t raw_at = (half * 2 + (raw_row >> 6)) * (C::RAW / 4) + (raw_row & 63) * 128;
    // Operands that take no 16-byte copies: an element of each of 32 rows a lane, neighbours side by side, into this warp's own part
    // of the ring's memory, from where a lane reads its row: 32-bit ones by copies of 4 bytes a chunk ahead, 16-bit ones through
    // registers. (A lane that reads its row from memory asks for 32 lines an instruction, 4 us a chunk.)
    constexpr int PITCH = 36, BUFFERS = sizeof(TI) == 4 ? 2 : 1;
    TI* mine = reinterpret_cast<TI*>(smem) + cw * BUFFERS * 32 * PITCH;
    static_assert(C::A_WARPS * BUFFERS * 32 * PITCH * 4 <= C::RAWS * C::RAW, "the warps' parts of the ring's memory");
    TI held[VEC || BUFFERS == 2 ? 1 : 32];
    auto fetch = [&](int c, int buffer) {
      const int k = c * CHUNK + half * 32 + lane;
      const bool there = k < p.K;
#pragma unroll
      for (int r = 0; r < 32 && c < last; ++r) {  // (behind the last chunk nothing: the sums are put where it would land)
        const int n = min(dual ? n0 + quarter * 16 + (r & 15) : n0 + quarter * 32 + r, p.N - 1);
        const TI* src = (const TI*)p.W + (there ? (size_t)(dual && (r & 16) ? p.N + n : n) * p.K + k : 0);
        if constexpr (BUFFERS == 2) cp_async4(mine + (buffer * 32 + r) * PITCH + lane, src, there);
        else held[r] = there ? __ldg(src) : TI(0.f);
      }
      if (BUFFERS == 2) asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t a_at = tmem + ((uint32_t)(quarter * 32) << 16) + C::A_AT + half * 16;
    typename C::RowMarks marks;
    if constexpr (!VEC) {
      pdl_wait();
      fetch(first + set, 0);
    }
    for (int c = first + set, n = set, buffer = 0; c < last; c += C::SETS, n += C::SETS, buffer ^= BUFFERS - 1) {
      const int st = n % C::STAGES, raw = n % C::RAWS;
      uint32_t w[C::P][16];
      if constexpr (VEC) {
        if (!warp_wait(&raw_full[raw], (n / C::RAWS) & 1, p.err, abort_flag)) break;
        const uint8_t* src = smem + raw * C::RAW + raw_at;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          uint2 x[C::P];
          split(x, *reinterpret_cast<const float4*>(src + ((q ^ (raw_row & 7)) << 4)), marks);
#pragma unroll
          for (int t = 0; t < C::P; ++t) w[t][2 * q] = x[t].x, w[t][2 * q + 1] = x[t].y;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[raw]);
      } else {
        if constexpr (BUFFERS == 2) {
          fetch(c + C::SETS, buffer ^ 1);
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          __syncwarp();
        } else {
#pragma unroll
          for (int r = 0; r < 32; ++r) mine[r * PITCH + lane] = held[r];
          __syncwarp();
          fetch(c + C::SETS, 0);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          uint2 x[C::P];
          split(x, *reinterpret_cast<const decltype(load4<false>((const TI*)p.W, 0))*>(mine + (buffer * 32 + lane) * PITCH + 4 * q), marks);
#pragma unroll
          for (int t = 0; t < C::P; ++t) w[t][2 * q] = x[t].x, w[t][2 * q + 1] = x[t].y;
        }
      }
      if (!warp_wait(&done[st], ((n / C::STAGES) & 1) ^ 1, p.err, abort_flag)) break;
      tc_fence_after();
#pragma unroll
      for (int t = 0; t < C::P; ++t) tmem_st16(a_at + st * C::A_COLS + t * CHUNK / 2, w[t]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[st]);
    }
    if (!VEC && BUFFERS == 2) asm volatile("cp.async.wait_all;" ::: "memory");
    if (C::P == 3) note(&row_marks[l], marks.word());
  } else {
    // ---- sums: thread = weight row, COLS tokens
    const int quarter = warp & 3, col0 = (warp >> 2) * C::COLS;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + col0, total = lane_base + C::SUM_AT;
    float sum[C::COLS];
    bool ok = true;
    auto add_up = [&](uint32_t at, bool starts) {
#pragma unroll
      for (int j = 0; j < C::COLS; j += 16) {
        uint32_t x[16];
        tmem_ld16_async(at + j, x);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 16; ++q) sum[j + q] = starts ? __uint_as_float(x[q]) : sum[j + q] + __uint_as_float(x[q]);
      }
      tc_fence_before();
      __syncwarp();
    };
    for (int c = first, i = 0; c < last; ++c, ++i) {
      const bool begins = i % BLOCK == 0, ends = i % BLOCK == BLOCK - 1 || c == last - 1, more = p.slices == 1 && i >= BLOCK;
      if (C::P == 3 && ends) {
        ok = warp_wait(small_full, (i / BLOCK) & 1, p.err, abort_flag);
        if (!ok) break;
        tc_fence_after();
        add_up(lane_base + C::SMALL_AT, begins);
        if (lane == 0) mbar_arrive(small_empty);
      }
      ok = warp_wait(&done[i % C::STAGES], (i / C::STAGES) & 1, p.err, abort_flag);
      if (!ok) break;
      tc_fence_after();
      add_up(lane_base + (i & 1) * NT, begins && !(C::P == 3 && ends));
      if (lane == 0) mbar_arrive(&acc_empty[i & 1]);
      if (ends && C::SUM_IN_SMEM) {
        float* mine = total_s + col0 * ROWS + quarter * 32 + lane;
#pragma unroll
        for (int j = 0; j < C::COLS; ++j) mine[j * ROWS] = more ? mine[j * ROWS] + sum[j] : sum[j];
      } else if (ends) {
        const uint32_t at = total + (p.slices > 1 ? i / BLOCK * NT : 0);
#pragma unroll
        for (int j = 0; j < C::COLS; j += 16) {
          if (more) {
            uint32_t x[16];
            tmem_ld16_async(at + j, x);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 16; ++q) sum[j + q] = __uint_as_float(x[q]) + sum[j + q];
          }
          if (c < last - 1) tmem_st16(at + j, reinterpret_cast<const uint32_t*>(sum + j));
        }
        tmem_st_wait();
      }
    }
    if (ok && !C::SUM_IN_SMEM) {
      // [block][token][row]; every contraction is done, so the stages are free
      float* mine = reinterpret_cast<float*>(smem) + col0 * ROWS + quarter * 32 + lane;
      const int held = p.slices > 1 ? (last - first - 1) / BLOCK : 0;
#pragma unroll 1
      for (int b = 0; b < held; ++b)
#pragma unroll 1
        for (int j = 0; j < C::COLS; j += 16) {
          float v[16];
          tmem_ld16(total + b * NT + j, v);
#pragma unroll
          for (int q = 0; q < 16; ++q) mine[(size_t)(b * NT + j + q) * ROWS] = v[q];
        }
#pragma unroll
      for (int j = 0; j < C::COLS; ++j) mine[(size_t)(held * NT + j) * ROWS] = sum[j];
    }
  }
  // ---- results: every thread, in one short loop (unrolled per accumulator column its code came from L2, at 290 clocks a
  // column); the CTAs of a cluster share the tile's outputs and read each other's sums
  __syncwarp();
  pdl_wait();
  if (p.slices > 1) cluster_sync_all();
  else __syncthreads();
  const int items = *abort_flag ? 0 : OUTS * min(NT, p.M - m0);
  uint32_t some_lossy = 0;  // (a CTA a lane)
  if (C::P == 3) some_lossy = p.slices == 1 ? *any_lossy : ld_cluster_u32(smem_u32(any_lossy), lane % p.slices, 0);
  // a row's marks in all of K
  auto marks_of = [&](const uint32_t* at) {
    uint32_t word = *at;
    if (p.slices > 1)
      for (int s = 0; s < p.slices; ++s) word |= ld_cluster_u32(smem_u32(at), s, 0);
    return word;
  };
#pragma unroll 1
  for (int e0 = rank * C::THREADS; e0 < items; e0 += p.slices * C::THREADS) {
    const int e = e0 + threadIdx.x, o = e % OUTS, m = e / OUTS, n = n0 + o;
    const bool live = e < items && n < p.N;
    const int row = dual ? (o >> 4) * 32 + (o & 15) : o;
    float v = 0.f, u = 0.f;
    if (live && p.slices == 1) {
      const float* sums = (C::SUM_IN_SMEM ? total_s : reinterpret_cast<const float*>(smem)) + (size_t)m * ROWS + row;
      v = sums[0];
      if (dual) u = sums[16];
    } else if (live) {
      // eight blocks' sums in flight at once, whichever CTA holds them: one CTA's after the other took a round trip each
      int s = 0, from = 0, to = blocks / p.slices;
#pragma unroll 1
      for (int b0 = 0; b0 < blocks; b0 += 8) {
        float x[8], y[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          if (b0 + b >= blocks) break;
          if (b0 + b == to) {
            from = to;
            ++s;
            to = (s + 1) * blocks / p.slices;
          }
          const uint32_t at = (uint32_t)(((b0 + b - from) * NT + m) * ROWS + row) * 4;
          x[b] = ld_cluster(smem_u32(smem), s, at);
          if (dual) y[b] = ld_cluster(smem_u32(smem), s, at + 64);
        }
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          if (b0 + b >= blocks) break;
          v = b0 + b > 0 ? v + x[b] : x[b];
          if (dual) u = b0 + b > 0 ? u + y[b] : y[b];
        }
      }
    }
    uint32_t token = 0, weight = 0, up_weight = 0;
    if (__any_sync(0xffffffffu, some_lossy) && live) {
      token = marks_of(&token_marks[m]);
      weight = marks_of(&row_marks[row]);
      if (dual) up_weight = marks_of(&row_marks[row + 16]);
    }
    const bool again = live && !settled(v, token, weight), again_u = live && dual && !settled(u, token, up_weight);
    if (__any_sync(0xffffffffu, again || again_u)) {
      v = settle<TI>(p, v, again, m0 + m, n);
      if (dual) u = settle<TI>(p, u, again_u, m0 + m, p.N + n);
    }
    if (live) finish<TI>(p, m0 + m, n, v, u);
  }
  if (p.slices > 1) cluster_sync_all();  // no CTA leaves while another reads its sums
  if (*abort_flag) {
    // contractions and copies in flight end before their memory is given back
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 2000000ull) { }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

int scratch_ld(int K) { return (K + 7) / 8 * 8; }

template <typename TI, int NT, bool VEC>
int prepare() {
  using C = Form<TI, NT>;
  static const cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<TI, NT, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  CUCA_REQUIRE(e == cudaSuccess, "gemm: %d bytes of shared memory were refused: %s", C::SMEM, cudaGetErrorString(e));
  return 0;
}

template <typename TI, int NT, bool VEC>
int launch(GemmParams p, int slices, void* scratch, cudaStream_t stream) {
  using C = Form<TI, NT>;
  auto kernel = gemm_f32_kernel<TI, NT, VEC>;
  if (int rc = prepare<TI, NT, VEC>()) return rc;
  const bool dual = p.epilogue == EPI_SWIGLU;
  const int outs = dual ? ROWS / 2 : ROWS;
  p.tiles_m = (p.M + NT - 1) / NT;
  p.slices = slices;
  const long long ctas = (long long)p.tiles_m * ((p.N + outs - 1) / outs) * slices;
  CUCA_REQUIRE(ctas < (1ll << 31), "gemm: %d x %d outputs are too many", p.M, p.N);
  CUtensorMap tmW = {}, tmX = {};
  CUCA_REQUIRE(!VEC || cuca_tensor_map_2d(p.W, 4, (uint64_t)p.N * (dual ? 2 : 1), p.K, p.K, 64, &tmW), "gemm: weight tensor map failed");
  if (C::PRE) {
    const int ld = scratch_ld(p.K);
    CUCA_REQUIRE(scratch && ((uintptr_t)scratch & 15) == 0, "gemm: %d tokens need scratch", p.M);
    CUCA_REQUIRE(cuca_tensor_map_2d(scratch, 2, (uint64_t)C::P * p.M, p.K, ld, NT, &tmX), "gemm: tensor map of the tokens failed");
    uint16_t* marks = (uint16_t*)scratch + (size_t)C::P * p.M * ld;
    p.marks = marks;
    for (int m = 0; m < p.M; m += 65535)  // (the most rows of a launch)
      cuca_launch(split_kernel<TI, VEC>, dim3((p.K + SPLIT_RUN - 1) / SPLIT_RUN, std::min(p.M - m, 65535)), dim3(256), 0, stream, true,
                  (const TI*)p.A, (__nv_bfloat16*)scratch, marks, m, p.M, p.K, p.lda, ld);
  }
  if (slices > 1) cuca_launch_cluster(kernel, dim3((unsigned)ctas), dim3(C::THREADS), C::SMEM, stream, true, (unsigned)slices, tmW, tmX, p);
  else cuca_launch(kernel, dim3((unsigned)ctas), dim3(C::THREADS), C::SMEM, stream, true, tmW, tmX, p);
  return 0;
}

// How many clusters of `s` CTAs the device holds at once: a GPC's SMs rarely divide by 8.
template <typename TI, int NT, bool VEC>
int clusters_held(int s) {
  static int held[MAX_CLUSTER + 1] = {};  // (the same answer whoever asks first)
  if (!held[s]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s * cuca_device_sms());
    cfg.blockDim = dim3(Form<TI, NT>::THREADS);
    cfg.dynamicSmemBytes = Form<TI, NT>::SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = s;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (prepare<TI, NT, VEC>() || cudaOccupancyMaxActiveClusters(&n, gemm_f32_kernel<TI, NT, VEC>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = cuca_device_sms() / s / 2 + 1;
    }
    held[s] = n;
  }
  return held[s];
}

// Whether a cluster of `slices` CTAs can share K: each has blocks, and its tensor memory holds their sums.
template <typename TI, int NT>
bool holds(int K, int slices) {
  const int blocks = (K + CHUNK * BLOCK - 1) / (CHUNK * BLOCK);
  return slices == 1 || (slices > 1 && slices <= std::min(MAX_CLUSTER, blocks) && (blocks + slices - 1) / slices <= Form<TI, NT>::BLOCKS_HELD);
}

// The form with the least estimated time: rounds of CTAs times a CTA's chunks, whose cost in us (`chunk_us`) was measured as the
// slope over K, and a third more where narrow tiles of tokens read the same weights side by side; 3.5 us a launch, for a cluster
// 1.3 more and 0.15 for every block's sums that are read across it, 3 for the tokens' split. Measured, us: K = 8,192, 2,048 rows, one
// token: 1, 4, 6, 8 CTAs a tile 86, 30, 27, 41 (128 CTAs in clusters of eight do not fit at once); 24 tokens, tiles of 16 by 4 CTAs
// 37.2, of 32 by 6 30.5; K = 2,048, 64 tokens, tiles of 16 by 2 21.3, of 32 by 4 16.1, of 64 by 5 19.5.
struct Choice { int nt, slices; double cost; };
template <typename TI, int NT, bool VEC>
void consider(Choice& best, int M, int N, int K, bool dual, double chunk_us) {
  const int outs = dual ? ROWS / 2 : ROWS, blocks = (K + CHUNK * BLOCK - 1) / (CHUNK * BLOCK);
  const long long tiles = (long long)((M + NT - 1) / NT) * ((N + outs - 1) / outs);
  if (NT <= 32 && M > NT) chunk_us *= 1.3;
  for (int s = 1; s <= MAX_CLUSTER; ++s) {
    const int per = (blocks + s - 1) / s;
    if (!holds<TI, NT>(K, s) || (s > 1 && (per == (blocks + s - 2) / (s - 1) || tiles * (s - 1) >= cuca_device_sms()))) continue;
    const int held = s > 1 ? clusters_held<TI, NT, VEC>(s) : cuca_device_sms();
    const double cost = (double)((tiles + held - 1) / held) * (per * BLOCK * chunk_us + (s > 1 ? 4.8 + 0.15 * blocks : 3.5)) + (Form<TI, NT>::PRE ? 3. : 0.);
    if (cost < best.cost) best = {NT, s, cost};
  }
}
template <typename TI, bool VEC>
Choice choose(int M, int N, int K, bool dual) {
  Choice best = {0, 1, 1e30};
  consider<TI, 16, VEC>(best, M, N, K, dual, 0.64);
  if (M > 16) consider<TI, 32, VEC>(best, M, N, K, dual, 0.7);
  if (M > 32) consider<TI, 64, VEC>(best, M, N, K, dual, 0.92);
  if (M > 64) consider<TI, 96, VEC>(best, M, N, K, dual, 1.13);
  return best;
}

template <typename TI, bool VEC>
int go(const GemmParams& p, void* scratch, int form_tokens, int form_slices, cudaStream_t stream) {
  Choice f = {form_tokens, form_slices, 0.};
  if (!f.nt) f = choose<TI, VEC>(p.M, p.N, p.K, p.epilogue == EPI_SWIGLU);
#define FORM(NT)                                                                                           \
  if (f.nt == NT) {                                                                                        \
    CUCA_REQUIRE((holds<TI, NT>(p.K, f.slices)), "gemm: K = %d is not cut in %d this way", p.K, f.slices); \
    return launch<TI, NT, VEC>(p, f.slices, scratch, stream);                                              \
  }
  FORM(16)
  FORM(32)
  FORM(64)
  FORM(96)
#undef FORM
  CUCA_REQUIRE(false, "gemm: no tiles of %d tokens", f.nt);
}

}  // namespace

// Most tokens for which cuca_gemm_f32 needs no scratch. Beyond, for each token so many 16-bit values, the whole 16-byte aligned:
// its parts, three of 32-bit operands and one of 16-bit ones, each K rounded up to a multiple of 8, and its marks.
CUCA_API int cuca_gemm_f32_few_tokens() { return FEW_TOKENS; }
CUCA_API int cuca_gemm_f32_scratch_per_token(int in_dtype, int K) {
  return (in_dtype == CUCA_F32 ? 3 : 1) * scratch_ld(K) + (K + SPLIT_RUN - 1) / SPLIT_RUN;
}

// out = epilogue(A[M,K] W[N,K]^T). in_dtype: A, W and bias; out_dtype: out.
// epilogue 0 store, 1 out (32-bit) += result, 2 SwiGLU (W has 2N rows).
// form_tokens, form_slices: tokens of a tile (16, 32, 64, 96) and CTAs that share its K (1 to 8), 0: the library's choice.
CUCA_API int cuca_gemm_f32(const void* A, const void* W, const void* bias, void* out, int in_dtype, int out_dtype, int M,
                           int N, int K, int lda, int ldo, int epilogue, int* err, void* scratch, int form_tokens,
                           int form_slices, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  CUCA_REQUIRE(K > 0 && lda >= K && ldo >= N, "gemm: bad sizes M=%d N=%d K=%d lda=%d ldo=%d", M, N, K, lda, ldo);
  CUCA_REQUIRE(epilogue != EPI_RESIDUAL || out_dtype == CUCA_F32, "gemm: the residual stream is 32-bit");
  CUCA_REQUIRE(epilogue != EPI_SWIGLU || bias == nullptr, "gemm: SwiGLU takes no bias");
  CUCA_REQUIRE(epilogue >= EPI_STORE && epilogue <= EPI_SWIGLU, "gemm: unknown epilogue %d", epilogue);
  CUCA_REQUIRE((in_dtype == CUCA_F32 && out_dtype == CUCA_F32) || (in_dtype == CUCA_BF16 && (out_dtype == CUCA_F32 || out_dtype == CUCA_BF16)),
               "gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
  GemmParams p = {A, W, bias, out, err, M, N, K, lda, ldo, epilogue, out_dtype == CUCA_F32, nullptr, 0, 0};
  const bool vec = in_dtype == CUCA_F32 && K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  int rc;
  if (in_dtype == CUCA_BF16) rc = go<__nv_bfloat16, false>(p, scratch, form_tokens, form_slices, stream);
  else if (vec) rc = go<float, true>(p, scratch, form_tokens, form_slices, stream);
  else rc = go<float, false>(p, scratch, form_tokens, form_slices, stream);
  if (rc) return rc;
  CUCA_CHECK_LAUNCH("gemm_f32");
  return 0;
}
