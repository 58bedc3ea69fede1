// Attention of prompt portions over a cached latent on the 5th-generation tensor cores (bfloat16 cache, 32-bit scores and
// sums): see latent_attention_mma.cu, which keeps single tokens and the sizes that this form refuses.
//
// Every head attends over the same cached rows [c | k_rot] (Dk values, the first `rank` of them the "values"), so the 128
// rows of a contraction are TQ consecutive tokens of one request times HB heads, which see nearly the same keys. A CTA walks
// the keys in tiles of 64 positions:
//
//   S[128, 64]       = Q K^T     over Dk values; two score buffers, the scores one tile ahead of the softmax
//   O[128, columns] += P V       V the same tile in shared memory, P written as bf16 over the scores it came from
//
// The 512 columns of tensor memory do not hold 512 columns of O beside the scores, so a CTA takes half of them and
// makes the scores again: 1.3 times the arithmetic, no exchange between CTAs. The first 256 values of Q lie in tensor memory
// too, the rest in shared memory beside two key tiles (64 x 576 values: 72 KB each, 227 KB in all).
//
// Key tiles come page by page through the copy engine, those with keys outside the group's by 16-byte cp.async with zeros there;
// one warp issues contractions, whatever is ready first; eight warps own the rows, two threads a row. A tile takes 4,150
// clocks: 1,550 of scores and 520 of P V on the tensor pipe, and with two tiles' memory a tile's copies (2,500) start when the
// P V two tiles before is done. A CTA's start, 288 KB of 32-bit queries, is 15 us of some 40. 2,048 tokens, 16 heads, 512 + 64,
// window 1,024: 152 us (361 TFLOP/s); 16 tokens of a head a group on mma.sync 526.
#include "tcgen05.cuh"
#include <math.h>

namespace {

typedef __nv_bfloat16 bf16;
constexpr int ROWS = 128, KEYS = 64;
constexpr int Q_CHUNK = ROWS * 128, K_CHUNK = KEYS * 128;  // 64 values of every row
constexpr int Q_COLS = 128;                                // tensor memory for the first 256 values of Q
constexpr int MAX_DK = 576;  // (two tiles of it and the queries' rest fill shared memory)
constexpr int O_AT = 0, S_AT = 256, Q_AT = 384;            // columns of tensor memory
constexpr int SOFT_WARPS = 8, LOAD_WARPS = 4, MMA_WARP = SOFT_WARPS + LOAD_WARPS;
constexpr int NTHREADS = 32 * (MMA_WARP + 1);
constexpr int HALVES = ROWS * 2 * 4;                       // a float of both halves of every row
constexpr int OUT_PITCH = 36;                              // floats a row of 32 output columns on its way out

struct Params {
  const float* qk;  // [rows, H, Dk] 32-bit: per head [query carried into the latent space | rotated part]
  float* out;       // [rows, H, rank]
  const bf16* pool; // [n_blocks][bs][Dk]
  int n_blocks, bs;
  const int* positions;
  const int* seq_of_row;
  const int* tables;
  int table_stride;
  const int* tile_row0;
  const int* tile_nrows;
  int H, HB, rank;
  float scale_log2;
  int window;
  const float* sink;
  int parts;        // CTAs that share a group's output columns
  int tma;          // whole key tiles come through the copy engine
  int* err;
};

constexpr int OUT_BYTES = SOFT_WARPS * 32 * OUT_PITCH * 4;  // all results on their way out lie in the two key tiles' memory
// A key tile's memory: the tile, the first 256 values of the queries on their way, or half of the results, whatever is larger.
__host__ __device__ constexpr int tile_bytes_of(int Dk) {
  int bytes = Dk / 64 * K_CHUNK;
  const int queries = (Dk < 256 ? Dk / 64 : 4) * Q_CHUNK, results = OUT_BYTES / 2;
  if (queries > bytes) bytes = queries;
  if (results > bytes) bytes = results;
  return bytes;
}
static_assert(OUT_BYTES / 2 % 1024 == 0, "tiles start at multiples of 1024 bytes");
constexpr int smem_bytes(int Dk) {
  const int q_chunks = Dk / 64 > 4 ? Dk / 64 - 4 : 0;
  return q_chunks * Q_CHUNK + 2 * tile_bytes_of(Dk) + HALVES + 1024 + 128;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;  // 0: nothing is read and the 16 bytes become zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {  // when this thread's copies so far have landed
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// the two warps that hold the halves of 32 rows
__device__ __forceinline__ void soft_sync(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(4 + quarter) : "memory"); }
// The same, and whether both are well: a wait can run out in one of them alone, so they leave only by this vote, together.
// A warp that left on its own would leave the other at the barrier, which has no limit.
__device__ __forceinline__ bool soft_vote(int quarter, bool ok) {
  uint32_t both;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.b32 p, %2, 0;\nbar.red.and.pred q, %1, 64, p;\nselp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(both) : "r"(4 + quarter), "r"((uint32_t)ok) : "memory");
  return both != 0;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int CHUNKS>  // Dk / 64
__global__ void __launch_bounds__(NTHREADS, 1)
latent_attention_tc_kernel(const __grid_constant__ CUtensorMap tmK, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* q_s = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int chunks = CHUNKS, Dk = 64 * CHUNKS, q_chunks = chunks > 4 ? chunks - 4 : 0;
  uint8_t* kv_s = q_s + q_chunks * Q_CHUNK;
  constexpr int tile_bytes = tile_bytes_of(Dk);
  float* halves = (float*)(kv_s + 2 * tile_bytes);  // [2][ROWS]
  uint64_t* q_full = (uint64_t*)(halves + 2 * ROWS);
  uint64_t* kv_full = q_full + 1;   // [2]
  uint64_t* kv_empty = kv_full + 2; // [2]
  uint64_t* s_full = kv_empty + 2;  // [2]
  uint64_t* p_full = s_full + 2;    // P is in tensor memory and O is rescaled
  uint64_t* pv_done = p_full + 1;
  uint32_t* tmem_slot = (uint32_t*)(pv_done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  pdl_trigger();
  pdl_wait();
  const int tile = blockIdx.x, part = blockIdx.z;
  const int row0 = p.tile_row0[tile], TQ = ROWS / p.HB;
  const int nrows = min(p.tile_nrows[tile], TQ);
  const int seq = p.seq_of_row[row0];
  if (seq < 0 || nrows <= 0) return;  // (the same for every thread of the block)
  const int head0 = blockIdx.y * p.HB;
  const int P0 = p.positions[row0], Pmax = P0 + nrows - 1;
  const int lo = (p.window > 0 && P0 - (p.window - 1) > 0) ? P0 - (p.window - 1) : 0;
  const int first_key = lo / KEYS * KEYS, n_tiles = Pmax / KEYS - lo / KEYS + 1;
  const int* table = p.tables + (size_t)seq * p.table_stride;
  // this CTA's output columns: whole chunks of 64
  const int v_chunks = p.rank / 64, c_first = part * v_chunks / p.parts, c_last = (part + 1) * v_chunks / p.parts;
  const int cols = (c_last - c_first) * 64;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 32 * SOFT_WARPS);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&kv_full[s], 32 * LOAD_WARPS);
      mbar_init(&kv_empty[s], 1);
      mbar_init(&s_full[s], 1);
    }
    mbar_init(p_full, 32 * SOFT_WARPS);
    mbar_init(pv_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // The queries as bfloat16, by all but the contracting warp: row r of the group is token r / HB, head head0 + r % HB. The first
  // 256 values are staged in the second key tile's memory for the threads that put them into tensor memory.
  uint8_t* staged = kv_s + tile_bytes;
  auto stage_queries = [&]() {
    constexpr int quads = Dk / 4, PER = (quads + 31) / 32;
    for (int r0 = warp; r0 < ROWS; r0 += 4 * (SOFT_WARPS + LOAD_WARPS)) {
      // four rows at a time, so that a warp has 20 loads in flight
      float4 v[4][PER];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + i * (SOFT_WARPS + LOAD_WARPS), tok = r / p.HB;
        const float4* q = reinterpret_cast<const float4*>(p.qk + ((size_t)(row0 + tok) * p.H + head0 + r % p.HB) * Dk);
#pragma unroll
        for (int n = 0; n < PER; ++n) {
          v[i][n] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < ROWS && tok < nrows && lane + 32 * n < quads) v[i][n] = __ldg(q + lane + 32 * n);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + i * (SOFT_WARPS + LOAD_WARPS);
#pragma unroll
        for (int n = 0; n < PER; ++n) {
          const int e = lane + 32 * n, c = e >> 4, unit = (e >> 1) & 7;  // 16 quads a chunk, two a 16-byte unit
          if (r < ROWS && e < quads)
            *reinterpret_cast<uint2*>((c < 4 ? staged + c * Q_CHUNK : q_s + (c - 4) * Q_CHUNK) + r * 128 + ((unit ^ (r & 7)) << 4) + (e & 1) * 8) =
                make_uint2(pack_bf16(v[i][n].x, v[i][n].y), pack_bf16(v[i][n].z, v[i][n].w));
        }
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * (SOFT_WARPS + LOAD_WARPS)) : "memory");
  };

  if (warp == MMA_WARP) {
    // ---- contractions (the whole warp walks the tiles, see elect_one)
    const uint32_t idesc_pv = instr_desc_b(true, cols);
    const uint64_t qd = smem_desc(smem_u32(q_s));
    auto ready = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)); };
    bool ok = warp_wait(q_full, 0, p.err, abort_flag);
    int next_sc = 0, next_pv = 0;
    unsigned spins = 0;
    unsigned long long idle_since = 0;
    // whatever is ready: the scores of tile t need its keys, and P of tile t - 2 to have left their buffer
    while (ok && next_pv < n_tiles) {
      bool progressed = false;
      if (next_sc < n_tiles && next_sc <= next_pv + 1 && ready(&kv_full[next_sc & 1], (next_sc >> 1) & 1)) {
        const int t = next_sc;
        fence_proxy_async();  // the copies' writes (and the queries') to the tensor cores
        tc_fence_after();
        const uint32_t acc = tmem + S_AT + (t & 1) * KEYS;
        const uint64_t kd = smem_desc(smem_u32(kv_s + (t & 1) * tile_bytes));
        if (elect_one()) {
#pragma unroll
          for (int c = 0; c < chunks; ++c) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint64_t b = kd + (uint64_t)((c * K_CHUNK + k * 32) >> 4);
              if (c < 4) umma_bf16_tmem_a(acc, tmem + Q_AT + c * 32 + k * 8, b, instr_desc(KEYS), c > 0 || k > 0);
              else umma_bf16(acc, qd + (uint64_t)(((c - 4) * Q_CHUNK + k * 32) >> 4), b, instr_desc(KEYS), 1);
            }
          }
          umma_commit(&s_full[t & 1]);
        }
        __syncwarp();
        ++next_sc;
        progressed = true;
      }
      if (next_pv < next_sc && ready(p_full, next_pv & 1)) {
        const int j = next_pv;
        tc_fence_after();
        const uint64_t vd = desc_mnmajor(smem_u32(kv_s + (j & 1) * tile_bytes + c_first * K_CHUNK), K_CHUNK, 1024);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < KEYS / 16; ++k)
            umma_bf16_tmem_a(tmem + O_AT, tmem + S_AT + (j & 1) * KEYS + k * 8, vd + (uint64_t)((k * 2048) >> 4), idesc_pv, j > 0 || k > 0);
          umma_commit(&kv_empty[j & 1]);
          umma_commit(pv_done);
        }
        __syncwarp();
        ++next_pv;
        progressed = true;
      }
      if (progressed) {
        idle_since = 0;
      } else if ((++spins & 63u) == 0) {
        if (__any_sync(0xffffffffu, *abort_flag)) break;
        const unsigned long long now = __shfl_sync(0xffffffffu, global_ns(), 0);
        if (idle_since == 0) {
          idle_since = now;
        } else if (now - idle_since > WAIT_LIMIT_NS) {
          if (p.err && lane == 0) atomicExch(p.err, CUCA_ERR_WAIT_TIMEOUT);
          *abort_flag = 1;
          break;
        }
      }
    }
  } else if (warp >= SOFT_WARPS) {
    // ---- key tiles: page by page through the copy engine; a tile with keys outside the group's by these threads, eight a key,
    // 16 bytes each, with zeros there
    const int tid = threadIdx.x - 32 * SOFT_WARPS, piece = tid & 7;
    auto load_tile = [&](int t) {
      uint8_t* tile = kv_s + (t & 1) * tile_bytes;
      const int key0 = first_key + t * KEYS;
      if (p.tma && key0 >= lo && key0 + KEYS - 1 <= Pmax) {
        if (tid == 0) mbar_expect_tx(&kv_full[t & 1], chunks * K_CHUNK);
        // one copy a thread, dealt to the warps in turn: a lane's copy takes 70 clocks to issue
        const int copy = lane * LOAD_WARPS + warp - SOFT_WARPS, c = copy % chunks, page = copy / chunks;
        if (page * p.bs < KEYS) {
          int blk = table[(key0 + page * p.bs) / p.bs];
          if (blk < 0 || blk >= p.n_blocks) {
            if (p.err) atomicExch(p.err, CUCA_ERR_BLOCK_RANGE);
            blk = 0;
          }
          tma_load_2d(tile + c * K_CHUNK + page * p.bs * 128, &tmK, &kv_full[t & 1], c * 64, blk * p.bs);
        }
        if (tid != 0) mbar_arrive(&kv_full[t & 1]);
        return;
      }
#pragma unroll
      for (int i = 0; i < KEYS / 16; ++i) {
        const int j = tid / 8 + 16 * i, kp = key0 + j;
        bool valid = kp >= lo && kp <= Pmax;
        const bf16* src = p.pool;
        if (valid) {
          const int blk = table[kp / p.bs];
          if (blk < 0 || blk >= p.n_blocks) {
            if (p.err) atomicExch(p.err, CUCA_ERR_BLOCK_RANGE);
            valid = false;
          } else {
            src += ((size_t)blk * p.bs + kp % p.bs) * Dk;
          }
        }
        const uint32_t at = smem_u32(tile) + j * 128 + ((piece ^ (j & 7)) << 4);
#pragma unroll
        for (int c = 0; c < chunks; ++c) cp_async16(at + c * K_CHUNK, valid ? src + c * 64 + piece * 8 : p.pool, valid);
      }
      cp_async_arrive(&kv_full[t & 1]);
    };
    load_tile(0);
    stage_queries();
    if (n_tiles > 1) {
      // (the queries' staging lay in the second tile's memory: read by all before, and written by generic stores)
      asm volatile("bar.sync 2, %0;" ::"n"(32 * (SOFT_WARPS + LOAD_WARPS)) : "memory");
      fence_proxy_async();
      load_tile(1);
    } else {
      asm volatile("bar.sync 2, %0;" ::"n"(32 * (SOFT_WARPS + LOAD_WARPS)) : "memory");
    }
    for (int t = 2; t < n_tiles; ++t) {
      if (!warp_wait(&kv_empty[t & 1], ((t >> 1) & 1) ^ 1, p.err, abort_flag)) break;
      load_tile(t);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---- two threads a row, 32 keys of a tile and half of the output columns each: first the queries into tensor memory
    const int quarter = warp & 3, half = warp >> 2;
    const int r = quarter * 32 + lane, tok = r / p.HB;
    const uint32_t lane_bits = (uint32_t)(quarter * 32) << 16;
    const bool row_ok = tok < nrows;
    const int row_pos = P0 + tok;
    const int row_lo = (p.window > 0 && row_pos - (p.window - 1) > 0) ? row_pos - (p.window - 1) : 0;
    stage_queries();
#pragma unroll 1
    for (int c = half; c < (chunks < 4 ? chunks : 4); c += 2) {
      uint32_t w[32];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<uint4*>(w + 4 * u) = *reinterpret_cast<const uint4*>(staged + c * Q_CHUNK + r * 128 + ((u ^ (r & 7)) << 4));
      tmem_st32_raw(tmem + lane_bits + Q_AT + c * 32, w);
    }
    asm volatile("bar.sync 2, %0;" ::"n"(32 * (SOFT_WARPS + LOAD_WARPS)) : "memory");  // the staging memory is free
    tmem_st_wait();
    tc_fence_before();
    mbar_arrive(q_full);
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      const uint32_t s_at = tmem + lane_bits + S_AT + (j & 1) * KEYS;
      ok = ok && warp_wait(&s_full[j & 1], (j >> 1) & 1, p.err, abort_flag);
      tc_fence_after();
      const int key0 = first_key + j * KEYS;
      uint32_t raw[32];
      tmem_ld32_nowait(s_at + half * 32, raw);
      tmem_ld_wait();
      // scores that every row of the group sees go without tests
      const bool whole = nrows == TQ && key0 + KEYS - 1 <= P0 && (p.window <= 0 || key0 >= Pmax - (p.window - 1));
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (!whole) {
          const int kp = key0 + half * 32 + i;
          if (!(row_ok && kp <= row_pos && kp >= row_lo)) raw[i] = 0xff800000u;  // -inf
        }
        mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(raw[i]));
      }
      // the other half's maximum; behind the barrier both halves have read their scores, so P may take their place
      halves[half * ROWS + r] = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      ok = soft_vote(quarter, ok);
      if (!ok) break;
      const float mx = fmaxf(halves[r], halves[ROWS + r]) * p.scale_log2;
      soft_sync(quarter);  // (both have read before either writes the next tile's)
      // The reference only moves when the maximum exceeds it by more than 8 (in log2 units): values up to 2^8 above it are
      // as exact in 32-bit sums and in bfloat16, and O is rescaled far less often.
      float m_new = m;
      if (mx > m + 8.f || m == -INFINITY) m_new = fmaxf(m, mx);
      const float corr = (m_new == -INFINITY || m == m_new) ? 1.f : fast_exp2(m - m_new);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), neg_m2 = make_float2(-m_use, -m_use);
      uint32_t pw[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float2 x2 = __ffma2_rn(make_float2(__uint_as_float(raw[2 * e]), __uint_as_float(raw[2 * e + 1])), scale2, neg_m2);
        const float2 p2 = make_float2(fast_exp2(x2.x), fast_exp2(x2.y));
        sum2[e & 1] = __fadd2_rn(sum2[e & 1], p2);
        pw[e] = pack_bf16(p2.x, p2.y);
      }
      tmem_st16(s_at + half * 16, pw);
      l = l * corr + (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
      m = m_new;
      // the P V before this one has finished before O is rescaled (its phase is awaited every time, so that the barrier never
      // runs two phases ahead of its waiters)
      if (j > 0) {
        ok = warp_wait(pv_done, (j - 1) & 1, p.err, abort_flag);
        if (!ok) continue;  // (to the next vote)
        tc_fence_after();
        if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll 1
          for (int c = half * 32; c < cols; c += 64) {
            float o[32];
            tmem_ld32(tmem + lane_bits + O_AT + c, o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= corr;
            tmem_st32(tmem + lane_bits + O_AT + c, o);
          }
        }
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(p_full);
    }
    ok = ok && warp_wait(pv_done, (n_tiles - 1) & 1, p.err, abort_flag);
    halves[half * ROWS + r] = l;
    ok = soft_vote(quarter, ok);
    if (ok) {
      tc_fence_after();
      l = halves[r] + halves[ROWS + r];
      if (p.sink && m != -INFINITY) l += fast_exp2(p.sink[head0 + r % p.HB] * 1.4426950408889634f - m);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      // every contraction is done, so the key tiles' memory is free: 32 columns at a time through this warp's share of it, so
      // that eight lanes store 128 bytes of a row
      float* mine = reinterpret_cast<float*>(kv_s) + warp * 32 * OUT_PITCH;
#pragma unroll 1
      for (int c = half * 32; c < cols; c += 64) {
        float o[32];
        tmem_ld32(tmem + lane_bits + O_AT + c, o);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<float4*>(mine + lane * OUT_PITCH + 4 * i) =
              make_float4(o[4 * i] * inv, o[4 * i + 1] * inv, o[4 * i + 2] * inv, o[4 * i + 3] * inv);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = i * 4 + lane / 8, row = quarter * 32 + rr, tk = row / p.HB;
          if (tk < nrows)
            *reinterpret_cast<float4*>(p.out + ((size_t)(row0 + tk) * p.H + head0 + row % p.HB) * p.rank + c_first * 64 + c + lane % 8 * 4) =
                *reinterpret_cast<const float4*>(mine + rr * OUT_PITCH + lane % 8 * 4);
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  if (*abort_flag) {
    // contractions in flight end before their memory is given back
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 2000000ull) { }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

template <int CHUNKS>
int launch(const CUtensorMap& tmK, const Params& p, int n_groups, cudaStream_t stream) {
  constexpr int smem = smem_bytes(64 * CHUNKS);
  static_assert(smem <= 227 * 1024, "shared memory");
  static const cudaError_t e = cudaFuncSetAttribute(latent_attention_tc_kernel<CHUNKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  CUCA_REQUIRE(e == cudaSuccess, "latent_attention_tc: %d bytes of shared memory were refused: %s", smem, cudaGetErrorString(e));
  cuca_launch(latent_attention_tc_kernel<CHUNKS>, dim3(n_groups, p.H / p.HB, p.parts), dim3(NTHREADS), smem, stream, true, tmK, p);
  CUCA_CHECK_LAUNCH("latent_attention_tc");
  return 0;
}

}  // namespace

// Tokens of a portion that one group of the tcgen05 form takes, 0 if it refuses the sizes: Dk and rank multiples of 64, Dk up
// to 576, rank from 64 to 512, heads a multiple of 8.
CUCA_API int cuca_latent_attention_tc_tokens(int H, int rank, int Dk) {
  if (H <= 0 || H % 8 != 0 || Dk % 64 != 0 || Dk > MAX_DK || rank % 64 != 0 || rank < 64 || rank > 512 || rank > Dk) return 0;
  return ROWS / (H % 16 == 0 ? 16 : 8);
}

// Group i: rows tile_row0[i] .. +tile_nrows[i]-1, up to cuca_latent_attention_tc_tokens consecutive rows of one request.
CUCA_API int cuca_latent_attention_tc(const float* qk, float* out, const void* pool, int n_blocks, int bs, const int* positions,
                                      const int* seq_of_row, const int* tables, int table_stride, const int* tile_row0,
                                      const int* tile_nrows, int n_groups, int H, int rank, int Dk, float scale, int window,
                                      const float* sink, int* err, cudaStream_t stream) {
  if (n_groups == 0) return 0;
  const int tokens = cuca_latent_attention_tc_tokens(H, rank, Dk);
  CUCA_REQUIRE(tokens > 0, "latent_attention_tc: sizes H=%d rank=%d Dk=%d are not taken", H, rank, Dk);
  CUCA_REQUIRE((((uintptr_t)qk | (uintptr_t)out | (uintptr_t)pool) & 15) == 0, "latent_attention_tc: operands off 16 bytes");
  CUCA_REQUIRE(n_groups < (1 << 30) && H / (ROWS / tokens) <= 65535, "latent_attention_tc: too many groups or heads");
  CUCA_REQUIRE(scale > 0.f, "latent_attention_tc: scale %g", scale);
  Params p;
  p.qk = qk; p.out = out; p.pool = (const bf16*)pool; p.n_blocks = n_blocks; p.bs = bs; p.positions = positions;
  p.seq_of_row = seq_of_row; p.tables = tables; p.table_stride = table_stride; p.tile_row0 = tile_row0;
  p.tile_nrows = tile_nrows; p.H = H; p.HB = ROWS / tokens; p.rank = rank;
  p.scale_log2 = scale * 1.4426950408889634f; p.window = window; p.sink = sink; p.parts = rank > 256 ? 2 : 1; p.err = err;
  CUtensorMap tmK = {};
  p.tma = bs >= 8 && bs <= KEYS && (bs & (bs - 1)) == 0 && cuca_tensor_map_bf16(pool, (uint64_t)n_blocks * bs, Dk, Dk, bs, &tmK);
  switch (Dk / 64) {
    case 1: return launch<1>(tmK, p, n_groups, stream);
    case 2: return launch<2>(tmK, p, n_groups, stream);
    case 3: return launch<3>(tmK, p, n_groups, stream);
    case 4: return launch<4>(tmK, p, n_groups, stream);
    case 5: return launch<5>(tmK, p, n_groups, stream);
    case 6: return launch<6>(tmK, p, n_groups, stream);
    case 7: return launch<7>(tmK, p, n_groups, stream);
    case 8: return launch<8>(tmK, p, n_groups, stream);
    default: return launch<9>(tmK, p, n_groups, stream);
  }
}
