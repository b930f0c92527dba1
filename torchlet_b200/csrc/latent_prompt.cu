// Latent attention over whole prompts on the 5th-generation tensor cores (tcgen05), bfloat16.
//
// A portion of a prompt that has nothing cached before it sees only keys of the step itself, and then it pays to EXPAND
// them: with K_h = W_uk,h c and V_h = W_uv,h c as two products over all heads, a (query, key) pair costs a head dim + rot + v
// multiplications instead of the latent form's rank + rot + rank, and no product of a head's own is needed before or after
// (16 heads, 128 + 64 against keys of rank 512: 320 against 1,088).  Two kernels, the products between them being ordinary
// ones:
//
//   rows    a block a token: the queries with their rotated part in bfloat16, [head][D + 64] (zeros past the rotated
//           part's end), and the token's cache row apart: c [rank], k_rot [64];
//   attend  a CTA takes two tiles of 128 queries of one (request, head) and walks over the keys in tiles of 128, as
//           attention_tc.cu does over pages: loader warps for K (the head's own D columns and the rotated part, which all
//           heads share) and V by TMA, 128-byte swizzle; one MMA warp that issues, for each tile of queries in turn,
//           O += P V of the key tile before (P read from tensor memory) and S = Q K^T of this one; four softmax warps a
//           tile of queries, a thread a row.  Keys are double-buffered, values, whose product runs a tile behind, are not:
//           shared memory holds 224 KB at D 128, rot 64, V 128.
//
// One prompt of 2,048 tokens, 16 heads of 128 + 64, rank 512: rows 17, the two products 20, attention 47 us (0.46 PFLOP/s, at a
// softmax of 2.4 us a key tile) against 22 + 23 + 430 + 23 for the latent form with its two products a head.
// Numerics are those of attention_tc.cu: float32 scores, maximum, sum and accumulator, P rounded to bfloat16 before P V.
// Error against 64 bits at scores of standard deviation 0.3, 1 and 3 (2,048 tokens, 16 heads of 128 + 64): 2.73, 3.17, 4.90e-3 against
// 2.73, 3.23, 4.70e-3 of the latent form: rounded keys of 128 entries move a large score a little more than rounded queries of
// 512 do.  (Sums over the rounded P, as the latent form takes: 2.72, 3.16, 4.81e-3, for 44 -> 48 us; not taken.)  A value without a number
// reaches the tokens before it in its tile of 128, as in attention_tc.cu; other requests' never.
// Every mbarrier wait is bounded (tcgen05.cuh); a wait that gives up records a code that tl_latent_prompt_error() returns, and
// the CTA still runs to its end and frees its TMEM.
#include <math.h>
#include <string.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "tcgen05.cuh"

namespace {

using namespace tc;

constexpr int ROWS = 128;       // queries of a tile (UMMA M)
constexpr int QTILES = 2;       // tiles of queries a CTA
constexpr int KEYS = 128;       // keys a tile (UMMA N of S, K of P V)
constexpr int THREADS = 352;    // warps 0-3 softmax of tile 0, 4-7 of tile 1, 8 MMA, 9 and 10 loaders
constexpr int SLAB = ROWS * 128;  // bytes of a [128 rows][64 bf16] swizzled slab
constexpr float RESCALE_THRESHOLD = 8.f;  // log2 units

__device__ int g_error_word = 0;

struct Params {
  const int* req_indptr;
  const int* tile_req;
  const int* tile_row;  // first token of the CTA's tiles within its request
  __nv_bfloat16* out;   // [tokens][heads V]
  long long out_stride;
  int rot_steps;  // 16-wide slices of the rotated part
  float scale_log2;
};

// 2^x by the special-function unit (ex2.approx: 2 ulp; the result is rounded to bfloat16 anyway).
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared-memory descriptor of the MN-major operand V: a tile is one or two slabs (64 elements
// of the head each) of [128 keys][64 elements]; 8 keys form a 1024-byte swizzle atom (stride
// byte offset), the slabs are SLAB bytes apart (leading byte offset).
__device__ __forceinline__ uint64_t smem_desc_v(uint32_t saddr) {
  uint64_t desc = 0;
  desc |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  desc |= (uint64_t)(SLAB >> 4) << 16;
  desc |= (uint64_t)(1024 >> 4) << 32;
  desc |= (uint64_t)1 << 46;
  desc |= (uint64_t)2 << 61;
  return desc;
}

// D (+)= A B with A read from tensor memory: row i of A in lane i, two bfloat16 of
// consecutive k in each 32-bit column (16 k = 8 columns an instruction).
__device__ __forceinline__ void mma_bf16_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                                bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_st_32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// P = exp2(S * scale - m) of one row as bfloat16 pairs into tensor memory at ``tmem_p`` (64
// columns).  The row's sum of the unrounded P goes to sum_a + sum_b.
__device__ __forceinline__ void exp_and_store(const uint32_t (&v)[KEYS], float scale_log2, float neg_m, uint32_t tmem_p,
                                              float& sum_a, float& sum_b) {
#pragma unroll
  for (int c = 0; c < KEYS; c += 64) {
    uint32_t packed[32];
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
      const float xa = fmaf(__uint_as_float(v[c + i]), scale_log2, neg_m);
      const float xb = fmaf(__uint_as_float(v[c + i + 1]), scale_log2, neg_m);
      const float a = fast_exp2(xa), b = fast_exp2(xb);
      sum_a += a;
      sum_b += b;
      __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
      packed[i >> 1] = *reinterpret_cast<uint32_t*>(&h);
    }
    tmem_st_32(tmem_p + (c >> 1), packed);
  }
}

template <int D, int V>
__global__ void __launch_bounds__(THREADS, 1)
latent_prompt_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_rot, const __grid_constant__ CUtensorMap map_v, const Params p) {
  constexpr int K_SLABS = D / 64 + 1, V_SLABS = V / 64;
  constexpr int QK_BYTES = K_SLABS * SLAB, V_BYTES = V_SLABS * SLAB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* q_tiles = smem;                      // 2 tiles of queries
  uint8_t* k_tiles = smem + 2 * QK_BYTES;       // 2 stages
  uint8_t* v_tile = smem + 4 * QK_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_tile + V_BYTES);
  uint64_t* k_full = bars;        // [2 stages]
  uint64_t* k_empty = bars + 2;   // [2 stages]
  uint64_t* v_full = bars + 4;
  uint64_t* v_empty = bars + 5;
  uint64_t* s_full = bars + 6;    // [2 tiles]  S_X of the next key tile is in tensor memory
  uint64_t* p_full = bars + 8;    // [2 tiles]  (4 arrivals: one per softmax warp) P_X is written
  uint64_t* o_done = bars + 10;   // [2 tiles]  the last P_X V is done
  uint64_t* q_full = bars + 12;
  uint64_t* v_clean = bars + 13;  // value rows past the CTA's last key are cleared
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heads vary fastest over the grid: the CTAs that see the most keys (the caller lists those first) start first for all
  const int h = blockIdx.x;
  const int req = p.tile_req[blockIdx.y];
  const int tok0 = p.req_indptr[req], q_len = p.req_indptr[req + 1] - tok0;
  const int row0 = p.tile_row[blockIdx.y];
  int ends[QTILES];  // key tiles [0, end) that a tile of queries needs
#pragma unroll
  for (int x = 0; x < QTILES; ++x) {
    const int start = row0 + x * ROWS;
    ends[x] = start < q_len ? (min(q_len, start + ROWS) - 1) / KEYS + 1 : 0;
  }
  const int j_end = max(ends[0], ends[1]);
  // The last key tile may hold rows of the next request, whose weights are exactly 0; but 0 x NaN is NaN, so the V loader
  // clears them before the tensor core reads them.  (Rows past the step's last token are zero-filled by the copy.)
  const bool edge = j_end * KEYS > q_len;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1);
    }
    mbar_init(v_full, 1);
    mbar_init(v_empty, 1);
    mbar_init(q_full, 1);
    mbar_init(v_clean, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 8) {
    tmem_alloc<512>(tmem_slot);
    tmem_relinquish();
  }
  tl::pdl_wait();
  tl::pdl_launch_dependents();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 9) {
    // -------------------------------------------------------- loader of queries and keys
    if (lane == 0) mbar_expect_tx(q_full, QTILES * QK_BYTES);
    __syncwarp();
    if (lane < QTILES * K_SLABS)
      tma_load_2d(q_tiles + lane * SLAB, &map_q, q_full, h * (D + 64) + lane % K_SLABS * 64, tok0 + row0 + lane / K_SLABS * ROWS);
    for (int j = 0; j < j_end; ++j) {
      const int s = j & 1;
      mbar_wait(&k_empty[s], ((j >> 1) & 1) ^ 1, abort_flag, &g_error_word, 1);
      if (lane == 0) mbar_expect_tx(&k_full[s], QK_BYTES);
      __syncwarp();
      uint8_t* dst = k_tiles + s * QK_BYTES + lane * SLAB;
      if (lane < K_SLABS - 1) tma_load_2d(dst, &map_k, &k_full[s], h * D + lane * 64, tok0 + j * KEYS);
      else if (lane == K_SLABS - 1) tma_load_2d(dst, &map_rot, &k_full[s], 0, tok0 + j * KEYS);
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------------ loader of values
    for (int j = 0; j < j_end; ++j) {
      mbar_wait(v_empty, (j & 1) ^ 1, abort_flag, &g_error_word, 2);
      if (lane == 0) mbar_expect_tx(v_full, V_BYTES);
      __syncwarp();
      if (lane < V_SLABS) tma_load_2d(v_tile + lane * SLAB, &map_v, v_full, h * V + lane * 64, tok0 + j * KEYS);
      if (edge && j == j_end - 1) {
        mbar_wait(v_full, j & 1, abort_flag, &g_error_word, 10);  // the tile has landed
        for (int i = lane; i < KEYS * V_SLABS * 8; i += 32) {     // a key's row: 128 bytes in each slab
          const int k = i / (V_SLABS * 8);
          if (j * KEYS + k >= q_len)
            *reinterpret_cast<uint4*>(v_tile + ((i >> 3) % V_SLABS) * SLAB + k * 128 + (i & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async();  // the tensor core reads what these stores wrote
        __syncwarp();
        if (lane == 0) mbar_arrive(v_clean);
      }
    }
  } else if (warp == 8) {
    // --------------------------------------------------------------------- MMA
    // The whole warp walks the loop and waits; one elected lane issues.  A tile's P V and next S go out together, behind one
    // wait for its P; the tiles take turns, which keeps one in its softmax while the other's MMAs run.
    const uint32_t idesc_s = idesc_bf16_f32(ROWS, KEYS);
    const uint32_t idesc_o = idesc_bf16_f32(ROWS, V) | (1u << 16);  // B (V) MN-major
    const uint64_t q_desc[QTILES] = {smem_desc_sw128(smem_addr(q_tiles)), smem_desc_sw128(smem_addr(q_tiles + QK_BYTES))};
    const uint64_t k_desc[2] = {smem_desc_sw128(smem_addr(k_tiles)), smem_desc_sw128(smem_addr(k_tiles + QK_BYTES))};
    const uint64_t v_desc = smem_desc_v(smem_addr(v_tile));
    const int k_steps = D / 16 + p.rot_steps;
    mbar_wait(q_full, 0, abort_flag, &g_error_word, 4);
    // One step past the last key tile, for the P V that runs a tile behind
    for (int j = 0; j <= j_end; ++j) {
      if (j > 0) mbar_wait(v_full, (j - 1) & 1, abort_flag, &g_error_word, 6);
      if (edge && j == j_end) mbar_wait(v_clean, 0, abort_flag, &g_error_word, 11);
      if (j < j_end) mbar_wait(&k_full[j & 1], (j >> 1) & 1, abort_flag, &g_error_word, 3);
      const bool work_1 = j <= ends[1] && ends[1] > 0;  // (the second tile's queries need no fewer keys than the first's)
#pragma unroll
      for (int x = 0; x < QTILES; ++x) {
        const uint32_t tmem_s = tmem_base + x * KEYS;     // S_x, and P_x in its first 64 columns
        const uint32_t tmem_o = tmem_base + 256 + x * V;  // O_x
        const bool do_pv = j > 0 && j - 1 < ends[x];      // O_x (+)= P_x V of key tile j - 1
        const bool do_s = j < ends[x];                    // S_x = Q_x K^T of key tile j
        if (!do_pv && !do_s) continue;
        if (do_pv) mbar_wait(&p_full[x], (j - 1) & 1, abort_flag, &g_error_word, 5);
        fence_after_sync();
        if (elect_one()) {
          if (do_pv) {
#pragma unroll
            for (int k = 0; k < KEYS / 16; ++k)  // 16 keys: 8 columns of P, two 8-key atoms of V (2048 bytes)
              mma_bf16_a_tmem(tmem_o, tmem_s + k * 8, v_desc + (uint64_t)(k * (2048 >> 4)), idesc_o, j > 1 || k > 0);
            if (j == ends[x]) mma_commit(&o_done[x]);
          }
          if (do_s) {
            const uint64_t b_desc = (j & 1) ? k_desc[1] : k_desc[0];
#pragma unroll
            for (int k = 0; k < D / 16 + 4; ++k) {  // slab k / 4, 32 bytes a slice within its 128-byte rows
              const uint64_t offset = (uint64_t)(((k >> 2) * SLAB + (k & 3) * 32) >> 4);
              if (k < k_steps) mma_bf16(tmem_s, q_desc[x] + offset, b_desc + offset, idesc_s, k > 0);
            }
            mma_commit(&s_full[x]);
          }
          if (x == 1 || !work_1) {
            if (j < j_end) mma_commit(&k_empty[j & 1]);
            if (j > 0) mma_commit(v_empty);
          }
        }
        __syncwarp();
      }
    }
  } else {
    // ----------------------------------------------------------------- softmax
    const int x = warp >> 2, quarter = warp & 3;
    const int pos = row0 + x * ROWS + quarter * 32 + lane;  // row of the tile = lane of tensor memory
    const bool row_valid = pos < q_len;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tmem_s = tmem_base + x * KEYS + lane_base;
    const uint32_t tmem_o = tmem_base + 256 + x * V + lane_base;
    const int num_tiles = x == 0 ? ends[0] : ends[1];
    float m_ref = -INFINITY, l_sum = 0.f;  // m_ref in log2 units (already scaled)
    for (int t = 0; t < num_tiles; ++t) {
      const int key0 = t * KEYS;
      mbar_wait(&s_full[x], t & 1, abort_flag, &g_error_word, 7);
      fence_after_sync();
      uint32_t v[KEYS];  // the row of S, in registers
#pragma unroll
      for (int c = 0; c < KEYS; c += 32) tmem_ld_32(tmem_s + c, reinterpret_cast<uint32_t(&)[32]>(v[c]));
      tmem_ld_wait();
      // rows beyond the request's last (never stored) take whatever comes
      if (!__all_sync(0xffffffffu, !row_valid || key0 + KEYS - 1 <= pos)) {
#pragma unroll
        for (int i = 0; i < KEYS; ++i)
          if (key0 + i > pos) v[i] = __float_as_uint(-INFINITY);
      }
      float m_a = -INFINITY, m_b = -INFINITY, m_c = -INFINITY, m_d = -INFINITY;
#pragma unroll
      for (int i = 0; i < KEYS; i += 8) {
        m_a = max3(m_a, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
        m_b = max3(m_b, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
        m_c = max3(m_c, __uint_as_float(v[i + 4]), __uint_as_float(v[i + 5]));
        m_d = max3(m_d, __uint_as_float(v[i + 6]), __uint_as_float(v[i + 7]));
      }
      const float m_tile = fmaxf(fmaxf(m_a, m_b), fmaxf(m_c, m_d)) * p.scale_log2;  // the factor is positive
      // the reference max moves only when the row's max has grown past the threshold
      float factor = 1.f;
      bool rescale = false;
      if (m_tile > m_ref + RESCALE_THRESHOLD || (m_ref == -INFINITY && m_tile > -INFINITY)) {
        factor = m_ref == -INFINITY ? 0.f : fast_exp2(m_ref - m_tile);
        rescale = m_ref != -INFINITY;
        m_ref = m_tile;
      }
      l_sum *= factor;
      if (__any_sync(0xffffffffu, rescale)) {
        // O_x is at rest: the arrival of S_x covered the P_x V issued before it
#pragma unroll 1
        for (int c = 0; c < V; c += 32) {
          uint32_t o[32];
          tmem_ld_32(tmem_o + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
          tmem_st_32(tmem_o + c, o);
        }
      }
      // P = exp2(S * scale - m_ref) as bfloat16 pairs over the first half of S's columns; row sum
      const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
      float sum_a = 0.f, sum_b = 0.f;
      exp_and_store(v, p.scale_log2, neg_m, tmem_s, sum_a, sum_b);
      l_sum += sum_a + sum_b;
      tmem_st_wait();
      fence_before_sync();  // our tcgen05.ld/st of S, P and O are done
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[x]);
    }
    if (num_tiles > 0) {
      mbar_wait(&o_done[x], 0, abort_flag, &g_error_word, 9);
      fence_after_sync();
      const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
      __nv_bfloat16* dst = p.out + (size_t)(tok0 + (row_valid ? pos : 0)) * p.out_stride + (size_t)h * V;
#pragma unroll 1
      for (int c = 0; c < V; c += 32) {
        uint32_t o[32];
        tmem_ld_32(tmem_o + c, o);
        tmem_ld_wait();
        if (row_valid) {
          uint32_t packed[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
            packed[i >> 1] = *reinterpret_cast<uint32_t*>(&b);
          }
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)
            *reinterpret_cast<uint4*>(dst + c + 8 * q4) =
                make_uint4(packed[4 * q4], packed[4 * q4 + 1], packed[4 * q4 + 2], packed[4 * q4 + 3]);
        }
      }
    }
  }
  __syncwarp();
  fence_before_sync();
  __syncthreads();
  if (warp == 8) {
    fence_after_sync();
    tmem_dealloc<512>(tmem_base);
  }
}

// q: float32 rows of heads * (dim + rot_dim); queries: [T, heads (dim + 64)]; c: [T, rank]; k_rot: [T, 64].  dim, rank and
// rot_dim are even.
constexpr int ROW_THREADS = 256;
__global__ void __launch_bounds__(ROW_THREADS)
latent_prompt_rows_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ inv_freq,
                          const int* __restrict__ positions, const int* __restrict__ token_req, const int* __restrict__ block_table,
                          int table_width, const __nv_bfloat16* __restrict__ pages, int page_size, int num_pages,
                          __nv_bfloat16* __restrict__ queries, __nv_bfloat16* __restrict__ c, __nv_bfloat16* __restrict__ k_rot,
                          int heads, int dim, int rot_dim, int rot_dims, int rank) {
  tl::pdl_launch_dependents();
  __shared__ float turn[2][32];
  const int t = blockIdx.x, half = rot_dims / 2, width = dim + 64;
  const int pos = positions[t];
  if (threadIdx.x < half) sincosf((float)pos * inv_freq[threadIdx.x], &turn[0][threadIdx.x], &turn[1][threadIdx.x]);
  __syncthreads();
  tl::pdl_wait();
  const float* row = q + (size_t)t * q_stride;
  __nv_bfloat16* dst = queries + (size_t)t * heads * width;
  for (int e = threadIdx.x; e < heads * width / 2; e += ROW_THREADS) {
    const int h = e / (width / 2), i = (e - h * (width / 2)) * 2;
    const float* head = row + h * (dim + rot_dim);
    float out[2] = {0.f, 0.f};
    if (i < dim) {
      out[0] = head[i];
      out[1] = head[i + 1];
    } else {
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int r = i - dim + n;
        if (r >= rot_dim) continue;
        const float* rot = head + dim;
        float v = rot[r];
        if (r < half) v = v * turn[1][r] - rot[r + half] * turn[0][r];
        else if (r < rot_dims) v = v * turn[1][r - half] + rot[r - half] * turn[0][r - half];
        out[n] = v;
      }
    }
    *reinterpret_cast<__nv_bfloat162*>(dst + h * width + i) = __floats2bfloat162_rn(out[0], out[1]);
  }
  if (!TL_DEBUG_OK(pos >= 0 && pos / page_size < table_width, TL_DEBUG_POSITION, pos)) return;
  const int page = block_table[(size_t)token_req[t] * table_width + pos / page_size];
  if (!TL_DEBUG_OK(page >= 0 && page < num_pages, TL_DEBUG_PAGE, page)) return;
  const unsigned* kept = reinterpret_cast<const unsigned*>(pages + ((size_t)page * page_size + pos % page_size) * (rank + rot_dim));
  for (int i = threadIdx.x; i < rank / 2; i += ROW_THREADS) reinterpret_cast<unsigned*>(c + (size_t)t * rank)[i] = kept[i];
  if (threadIdx.x < 32)
    reinterpret_cast<unsigned*>(k_rot + (size_t)t * 64)[threadIdx.x] = 2 * threadIdx.x < rot_dim ? kept[rank / 2 + threadIdx.x] : 0u;
}

// ------------------------------------------------------------------ host side
struct MapKey {
  const void* base;
  uint64_t rows;
  uint32_t cols, box_rows;
  bool operator==(const MapKey& o) const { return base == o.base && rows == o.rows && cols == o.cols && box_rows == o.box_rows; }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    return ((reinterpret_cast<size_t>(k.base) * 1000003u ^ k.rows) * 1000003u ^ k.cols) * 1000003u ^ k.box_rows;
  }
};

bool cached_map(CUtensorMap* out, const void* base, uint64_t rows, uint32_t cols, uint32_t box_rows) {
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  static std::mutex lock;
  const MapKey key{base, rows, cols, box_rows};
  std::lock_guard<std::mutex> guard(lock);
  auto it = cache.find(key);
  if (it == cache.end()) {
    CUtensorMap map;
    if (!tc_host::make_map_bf16(&map, base, rows, cols, cols, box_rows)) return false;
    if (cache.size() > 1024) cache.clear();
    it = cache.emplace(key, map).first;
  }
  *out = it->second;
  return true;
}

template <int D, int V>
int launch(const CUtensorMap (&maps)[4], const Params& p, int heads, int tiles, cudaStream_t stream) {
  constexpr int SMEM = (4 * (D / 64 + 1) + V / 64) * SLAB + 1024 + 256;
  static_assert(SMEM <= 232448, "shared memory of one CTA");
  static const cudaError_t configured =
      cudaFuncSetAttribute(latent_prompt_kernel<D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (configured != cudaSuccess) return (int)configured;
  tl::launch_kernel(latent_prompt_kernel<D, V>, dim3(heads, tiles), THREADS, SMEM, stream, maps[0], maps[1], maps[2], maps[3], p);
  return TL_LAUNCH_CHECK();
}

}  // namespace

TL_DEBUG_READER(tl_latent_prompt_debug_error)

extern "C" {

int tl_latent_prompt_error() {
  int value = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&value, g_error_word, sizeof(int)) != cudaSuccess) return -1;
  if (value) cudaMemcpyToSymbol(g_error_word, &zero, sizeof(int));
  return value;
}

// Tokens of a request that a CTA takes.
int tl_latent_prompt_tokens() { return QTILES * ROWS; }

int tl_latent_prompt_rows(const float* q, int q_stride, const float* inv_freq, const int* positions, const int* token_req,
                          const int* block_table, int table_width, const void* pages, int page_size, int num_pages, void* queries,
                          void* c, void* k_rot, int tokens, int heads, int dim, int rot_dim, int rot_dims, int rank,
                          cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (dim % 2 || rank % 2 || rot_dim % 2 || rot_dim > 64 || rot_dims % 2 || rot_dims > rot_dim || heads <= 0 || page_size <= 0)
    return TL_ERR_UNSUPPORTED;
  tl::launch_kernel(latent_prompt_rows_kernel, tokens, ROW_THREADS, 0, stream, q, q_stride, inv_freq, positions, token_req, block_table,
                    table_width, (const __nv_bfloat16*)pages, page_size, num_pages, (__nv_bfloat16*)queries, (__nv_bfloat16*)c,
                    (__nv_bfloat16*)k_rot, heads, dim, rot_dim, rot_dims, rank);
  return TL_LAUNCH_CHECK();
}

// queries [tokens, heads (dim + 64)], keys [tokens, heads dim], k_rot [tokens, 64], values [tokens, heads vdim], out [tokens,
// heads vdim], all bfloat16.  tile_req / tile_row: request and first token (a multiple of tl_latent_prompt_tokens()) of each CTA;
// the tiles cover every request, none of which has cached tokens.  dim and vdim 64 or 128, rot_dim a multiple of 16 up to 64, at
// least 128 tokens.
int tl_latent_prompt(const void* queries, const void* keys, const void* k_rot, const void* values, const int* req_indptr,
                     const int* tile_req, const int* tile_row, int tiles, void* out, int tokens, int heads, int dim, int rot_dim,
                     int vdim, float scale, cudaStream_t stream) {
  if (tiles <= 0 || tokens <= 0) return 0;
  if ((dim != 64 && dim != 128) || (vdim != 64 && vdim != 128) || rot_dim <= 0 || rot_dim > 64 || rot_dim % 16 || heads <= 0 ||
      tiles > 65535 || tokens < KEYS || !(scale > 0.f))
    return TL_ERR_UNSUPPORTED;
  CUtensorMap maps[4];
  if (!cached_map(&maps[0], queries, tokens, heads * (dim + 64), ROWS) || !cached_map(&maps[1], keys, tokens, heads * dim, KEYS) ||
      !cached_map(&maps[2], k_rot, tokens, 64, KEYS) || !cached_map(&maps[3], values, tokens, heads * vdim, KEYS))
    return TL_ERR_UNSUPPORTED;
  const Params p{req_indptr, tile_req, tile_row, (__nv_bfloat16*)out, (long long)heads * vdim, rot_dim / 16, scale * 1.4426950408889634f};
  if (dim == 128) return vdim == 128 ? launch<128, 128>(maps, p, heads, tiles, stream) : launch<128, 64>(maps, p, heads, tiles, stream);
  return vdim == 128 ? launch<64, 128>(maps, p, heads, tiles, stream) : launch<64, 64>(maps, p, heads, tiles, stream);
}

}  // extern "C"
