// What the kernels share that walk a request's tokens with a matrix per head, [value columns, key channels] in 32-bit, held
// in registers.
#pragma once
#include "common.cuh"
#include "f32x2.cuh"

int cuca_device_sms();

namespace {

// An asynchronous copy of 4 or 16 bytes from global to shared memory.
__device__ __forceinline__ void cp_async_f(float* dst, const float* src, bool wide) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// How a scan block's 128 threads share the state: NS threads a run of NC neighbouring value columns, thread s of them the
// key channels 4 (s + NS i) .. + 3 for i < NR / 4 (neighbouring threads read neighbouring 16 bytes, of the state in memory
// and of a staged vector in shared memory). A thread reads NR values of every staged vector per token for NR NC state
// values: reading shared memory (128 bytes a clock and SM, whether lanes ask for the same words or not) is what limits
// few columns a thread, the shuffles of the sums over NS threads what limits few channels.
template <int NS_, int NR_, int NC_>
struct Split {
  static constexpr int NS = NS_, NR = NR_, NC = NC_, DP = NS * NR, PB = NC * 128 / NS, PAIRS = NR / 2;
  static constexpr int TC = DP <= 128 ? 16 : 2048 / DP;  // tokens staged at a time
  // tokens whose outputs are summed together: up to four, or up to eight
  static constexpr int U = NS / NC >= 4 ? 4 : NS / NC, U8 = NS / NC >= 8 ? 8 : U;
  static_assert(NC <= 4 && U >= 1, "a column's sum ends up with a thread of its own");
};

// The state rows of a thread, as pairs, from `st` (the first of its columns, d channels each) and back. vec: 16 bytes at
// a time. cols: how many of the NC columns there are.
template <typename C>
__device__ __forceinline__ void load_rows(f32x2 (&S)[C::NC][C::PAIRS], const float* st, int s, int d, int cols, int vec) {
#pragma unroll
  for (int c = 0; c < C::NC; ++c)
#pragma unroll
    for (int i = 0; i < C::NR / 4; ++i) {
      const int r = 4 * (s + C::NS * i);
      const float* at = st + (size_t)c * d + r;
      S[c][2 * i] = S[c][2 * i + 1] = 0;
      if (vec) {
        if (c < cols && r < d) f2_load4(at, S[c][2 * i], S[c][2 * i + 1]);
      } else {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = c < cols && r + j < d ? at[j] : 0.f;
        S[c][2 * i] = f2_pack(v[0], v[1]);
        S[c][2 * i + 1] = f2_pack(v[2], v[3]);
      }
    }
}
template <int NS, int PAIRS>
__device__ __forceinline__ void store_column(const f32x2 (&S)[PAIRS], float* st, int s, int d, int vec) {
#pragma unroll
  for (int i = 0; i < PAIRS / 2; ++i) {
    const int r = 4 * (s + NS * i);
    if (vec) {
      if (r < d) *reinterpret_cast<ulonglong2*>(st + r) = make_ulonglong2(S[2 * i], S[2 * i + 1]);
    } else {
      float v[4];
      f2_unpack(S[2 * i], v[0], v[1]);
      f2_unpack(S[2 * i + 1], v[2], v[3]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (r + j < d) st[r + j] = v[j];
    }
  }
}
template <typename C>
__device__ __forceinline__ void store_rows(const f32x2 (&S)[C::NC][C::PAIRS], float* st, int s, int d, int cols, int vec) {
#pragma unroll
  for (int c = 0; c < C::NC; ++c)
    if (c < cols) store_column<C::NS, C::PAIRS>(S[c], st + (size_t)c * d, s, d, vec);
}
// A thread's channels of a staged vector.
template <typename C>
__device__ __forceinline__ void staged_rows(f32x2 (&v)[C::PAIRS], const float* vec, int s) {
#pragma unroll
  for (int i = 0; i < C::NR / 4; ++i) f2_load4(vec + 4 * (s + C::NS * i), v[2 * i], v[2 * i + 1]);
}
// The values of a thread's columns, staged side by side (column `at`, a multiple of NC).
template <int NC>
__device__ __forceinline__ void staged_values(float (&v)[NC], const float* vec, int at) {
  if (NC == 4) {
    const float4 w = *reinterpret_cast<const float4*>(vec + at);
    v[0] = w.x; v[1 % NC] = w.y; v[2 % NC] = w.z; v[3 % NC] = w.w;
  } else if (NC == 2) {
    const float2 w = *reinterpret_cast<const float2*>(vec + at);
    v[0] = w.x; v[1 % NC] = w.y;
  } else {
    v[0] = vec[at];
  }
}
// A thread's part of a dot product over the channels: four partial sums.
template <int PAIRS>
__device__ __forceinline__ float dot_rows(const f32x2 (&a)[PAIRS], const f32x2 (&b)[PAIRS]) {
  f32x2 p = f2_mul(a[0], b[0]), q = f2_mul(a[1], b[1]);
#pragma unroll
  for (int i = 2; i < PAIRS; i += 2) {
    p = f2_fma(a[i], b[i], p);
    q = f2_fma(a[i + 1], b[i + 1], q);
  }
  return f2_sum4(p, q);
}
// The sums of N values (N a power of two, at most NS) over the NS threads of a run of columns: thread s gets the sum of
// value s / (NS / N). The first steps halve the number of values a thread is busy with, so N sums take hardly more
// shuffles, and no longer a chain of them, than one.
template <int NS, int N>
__device__ __forceinline__ float spread_sum(float (&v)[N], int s) {
  static_assert(N <= NS, "a thread a value");
  int stride = NS / 2;
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1, stride >>= 1) {
    const bool upper = s & stride;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, stride);
    }
  }
#pragma unroll
  for (int o = NS / N / 2; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

template <int N_> struct Count { static constexpr int value = N_; };

// Launches a scan of `smem` bytes of shared memory a block. A prompt's few blocks are to lie spread over the SMs: launched
// while the kernel before drains they would pile up on the SMs that come free first (measured on 128 blocks: twice the
// time), so such a launch asks for so much shared memory that no SM takes more than its share.
template <typename... KArgs, typename... Args>
int launch_blocks(const char* name, void (*kernel)(KArgs...), dim3 grid, int threads, int smem, cudaStream_t stream, Args... args) {
  const long long blocks = (long long)grid.x * grid.y * grid.z, sms = cuca_device_sms();
  const long long per_sm = (blocks + sms - 1) / sms;
  const int spread = per_sm <= 4 ? 228 * 1024 / ((int)per_sm + 1) + 1024 : 0;
  if (smem < spread) smem = spread;
  if (smem > 48 * 1024) {
    // The limit belongs to the kernel, not to the launch: one number for all launches, so that a smaller launch of another
    // thread cannot lower it between these two calls.
    constexpr int MOST = 128 * 1024;
    CUCA_REQUIRE(smem <= MOST, "%s: a block of %d bytes of shared memory is larger than %d", name, smem, MOST);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST);
    CUCA_REQUIRE(e == cudaSuccess, "%s: %d bytes of shared memory were refused: %s", name, smem, cudaGetErrorString(e));
  }
  cuca_launch(kernel, grid, dim3(threads), smem, stream, true, args...);
  CUCA_CHECK_LAUNCH(name);
  return 0;
}

// The same for a scan with `floats_per_token` floats of shared memory a token, twice over.
template <typename C, typename... KArgs, typename... Args>
int launch_scan(const char* name, void (*kernel)(KArgs...), int floats_per_token, int H, int n_seqs, int dv, cudaStream_t stream,
                Args... args) {
  return launch_blocks(name, kernel, dim3(H, n_seqs, (dv + C::PB - 1) / C::PB), 128, 2 * C::TC * floats_per_token * 4, stream,
                       args...);
}

}  // namespace
