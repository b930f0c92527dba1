// Plain CUDA-core matrix product  out[M, N] (+)= x[M, K] . w[N, K]^T + bias[N].
//
// This is the true 32-bit path (float operands, IEEE fused multiply-add, no tensor
// cores, no reduced-precision mode) and the any-size path for bfloat16 operands
// that the tensor-core kernels refuse.
//
// bfloat16 operands: each output element is the sum over k in ascending order.
//
// float32: every kernel here adds in the SAME order, which depends on K alone, so a row's result does not depend on
// which other rows are in the batch, nor on which kernel took it: K is cut into at most 16 pieces of
// piece_length(K) entries (a multiple of 32); a piece is an ascending chain of fused multiply-adds that starts
// at zero; four consecutive pieces are added in ascending order to a quarter, the quarters in ascending order to
// the result.  Sixteen short chains are what lets few rows' work be spread over the GPU, and their rounding errors
// are smaller than those of one chain of K.
//
//   gemm_f32_stream_kernel  few rows (M <= 32; narrow products up to 128): bound by reading the weights and, from 8 tokens
//       on, by the shared-memory reads of the products.  A warp takes 32 weight rows and up to 32 tokens; the warps of a block
//       take one piece (narrow products: the four blocks of a cluster take the quarters and add them through distributed
//       shared memory, so that 896 weight rows still give 112 blocks) or one quarter each (wide products), with weights and
//       tokens staged by cp.async in a ring of 32-entry chunks of the warp's own, so no warp waits for another.
//       8 tokens, K x N: 896 x 9728 10.3 us (3,420 GB/s), 4864 x 896 11.2 us, 896 x 896 4.1 us, 896 x 151936 106 us
//       (5,190 GB/s), one token there 85 us (6,400 GB/s); one 64 x 64 tile kernel took all of these before, where a decode
//       step of 8 tokens at 24 such layers spent 30 ms in its products and spends 1 now.
//   gemm_f32_tile_kernel    more rows: bound by the shared-memory reads of the 8 x 8 (or 8 x 4) register tile, two 16-byte
//       reads an operand and k for 64 products.  Where the tiles leave SMs idle, the four blocks of a cluster take a quarter
//       of K each.  509 tokens, K x N: 896 x 9728 212 us (42 TFLOP/s), 4864 x 896 148 us, 896 x 896 35 us; 42 TFLOP/s on the
//       largest products.
//   gemm_simt_kernel        any type, stride and alignment (the other two copy 16 bytes at a time, float32 alone).
//
// Reference counterparts: nn.Linear in v10_triton_paged_gqa/layer/gqa.py:122-124,84
// and model/qwen2_5.py:83-87; down_kernel / swiglu_kernel GEMMs in
// v10_triton_paged_gqa/kernel/ffn_swiglu.py:5-164.
#include <limits.h>

#include "common.cuh"

namespace {

using namespace tl;

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// Entries of a piece: a multiple of 32, so that at most 16 pieces cover K.
__host__ __device__ __forceinline__ int piece_length(int K) { return (K + 511) / 512 * 32; }

template <typename T, typename OutT, bool ACCUM>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const T* __restrict__ x, const T* __restrict__ w, const float* __restrict__ bias,
                 OutT* __restrict__ out, int M, int N, int K, int ldx, int ldw, int ldo) {
  tl::pdl_wait();               // everything before us in the stream is complete and visible
  tl::pdl_launch_dependents();  // the next kernel may start its own prologue

  constexpr bool PIECES = sizeof(T) == 4;
  __shared__ float xs[BK][BM + 1];
  __shared__ float ws[BK][BN + 1];
  __shared__ float totals[PIECES ? TM * TN : 1][256];  // of the quarters so far, a column a thread
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid % 16, ty = tid / 16;  // 16 x 16 threads, each TM x TN outputs
  float acc[TM][TN], quarter[PIECES ? TM : 1][TN];
  auto clear = [](auto& v) {
    for (auto& row : v)
#pragma unroll
      for (int j = 0; j < TN; ++j) row[j] = 0.f;
  };
  clear(acc);
  clear(quarter);
  // 64 rows x 16 k-values per operand, 4 per thread; the next step's are requested before this one's are multiplied
  T xr[4], wr[4];
  auto request = [&](int k0) {  // (past an edge the last entry; it is dropped below)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * 256, r = e / BK, k = min(k0 + e % BK, K - 1);
      xr[i] = x[(size_t)min(m0 + r, M - 1) * ldx + k];
      wr[i] = w[(size_t)min(n0 + r, N - 1) * ldw + k];
    }
  };
  const int piece_steps = PIECES ? piece_length(K) / BK : INT_MAX;
  int steps_left = piece_steps, pieces = 0;
  bool first_quarter = true;
  request(0);
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * 256, r = e / BK, c = e % BK;
      xs[c][r] = k0 + c < K && m0 + r < M ? to_float(xr[i]) : 0.f;
      ws[c][r] = k0 + c < K && n0 + r < N ? to_float(wr[i]) : 0.f;
    }
    __syncthreads();
    if (k0 + BK < K) request(k0 + BK);
#pragma unroll
    for (int c = 0; c < BK; ++c) {
      float xa[TM], wb[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) xa[i] = xs[c][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) wb[j] = ws[c][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(xa[i], wb[j], acc[i][j]);
    }
    __syncthreads();
    if constexpr (PIECES) {
      const bool last = k0 + BK >= K;
      if (--steps_left == 0 || last) {
        const bool quarter_ends = ++pieces == 4 || last;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            quarter[i][j] += acc[i][j];
            acc[i][j] = 0.f;
            if (quarter_ends) {
              const float sum = first_quarter ? quarter[i][j] : totals[i * TN + j][tid] + quarter[i][j];
              totals[i * TN + j][tid] = sum;
              quarter[i][j] = 0.f;
              if (last) acc[i][j] = sum;
            }
          }
        steps_left = piece_steps;
        if (quarter_ends) {
          first_quarter = false;
          pieces = 0;
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      OutT* o = out + (size_t)m * ldo + n;
      if (ACCUM)
        *o = from_float<OutT>(to_float(*o) + v);
      else
        *o = from_float<OutT>(v);
    }
  }
}

// ------------------------------------------------------------------------------------------ float32, 16-byte copies
__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes, zeros where ``live`` is false (nothing is read then).
__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(shared_address(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The float at ``p`` of this block's shared memory, read from block ``rank`` of the cluster.
__device__ __forceinline__ float peer_read(const float* p, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(shared_address(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void put(float* out, const float* bias, bool accum, int n, float v) {
  if (bias) v += bias[n];
  *out = accum ? *out + v : v;
}

constexpr int CHUNK = 32;       // k entries of a stage
constexpr int W_STRIDE = 36;    // floats a staged row takes: eight rows' 16 bytes lie in different banks
constexpr int STREAM_WARPS = 4;

template <int MT> constexpr int STREAM_STAGE = 32 * W_STRIDE + MT * W_STRIDE;  // floats
// A warp's lanes as TG token groups times 32 / TG row groups: a lane owns TG rows (row group + i 32 / TG) and MT / TG tokens
// (token group + j TG).  Every staged value then serves several products: one lane a row would read 9 times 16 bytes for 32
// products at 8 tokens and 33 for 128 at 32, this takes 6 and 12.
template <int MT> constexpr int TG = MT >= 8 ? 4 : (MT >= 4 ? 2 : 1);
// From 16 tokens on two stages, for more warps an SM: a warp requests its next chunk behind the products of this one and waits for
// it, the other warps' products cover the trip.  Three stages keep one more chunk on its way during the products.
template <int MT> constexpr int STREAM_STAGES = MT >= 16 ? 2 : 3;
template <int MT> constexpr int STREAM_SMEM = STREAM_WARPS * STREAM_STAGES<MT> * STREAM_STAGE<MT> * 4;

// One warp, 32 weight rows, the entries [k_begin, k_end) of K: ``end_piece`` is called after each piece with acc.
template <int MT, typename End>
__device__ __forceinline__ void stream_range(float* ring, const float* __restrict__ x, const float* __restrict__ w, int M,
                                             int N, int K, int ldx, int ldw, int n0, int k_begin, int k_end, int piece,
                                             float (&acc)[TG<MT>][MT / TG<MT>], End end_piece) {
  constexpr int STAGE = STREAM_STAGE<MT>, STAGES = STREAM_STAGES<MT>, G = TG<MT>;
  const int lane = threadIdx.x & 31;
  const int chunks = k_end > k_begin ? (k_end - k_begin + CHUNK - 1) / CHUNK : 0;
  const int seg = (lane & 7) * 4, row = lane >> 3;  // eight lanes a row of 128 bytes
  auto copy_w = [&](int c) {
    float* stage = ring + (c % STAGES) * STAGE;
    const int k = k_begin + c * CHUNK + seg;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = row + 4 * i;
      const bool live = n0 + r < N && k < K;
      copy16(stage + r * W_STRIDE + seg, live ? w + (size_t)(n0 + r) * ldw + k : w, live);
    }
  };
  auto copy_x = [&](int c) {
    float* stage = ring + (c % STAGES) * STAGE + 32 * W_STRIDE;
    const int k = k_begin + c * CHUNK + seg;
#pragma unroll
    for (int r = 0; r < MT; r += 4)
      if (MT >= 4 || row < MT) {
        const bool live = r + row < M && k < K;
        copy16(stage + (r + row) * W_STRIDE + seg, live ? x + (size_t)(r + row) * ldx + k : x, live);
      }
  };
  // the weights of the first stages are requested before the wait on the kernel that writes the tokens
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c)
    if (c < chunks) copy_w(c);
  tl::pdl_wait();
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c) {
    if (c < chunks) copy_x(c);
    copies_commit();  // (the weights' copies ride in the first group)
  }
  const int piece_chunks = piece / CHUNK;
  int in_piece = 0;
  for (int c = 0; c < chunks; ++c) {
    copies_wait<STAGES - 2>();
    __syncwarp();
    const float* stage = ring + (c % STAGES) * STAGE;
    const float* ws = stage + lane / G * W_STRIDE;
    const float* xs = stage + (32 + lane % G) * W_STRIDE;
#pragma unroll
    for (int k = 0; k < CHUNK; k += 4) {
      float4 wv[G];
#pragma unroll
      for (int i = 0; i < G; ++i) wv[i] = *reinterpret_cast<const float4*>(ws + i * (32 / G) * W_STRIDE + k);
#pragma unroll
      for (int j = 0; j < MT / G; ++j) {
        const float4 xv = *reinterpret_cast<const float4*>(xs + j * G * W_STRIDE + k);
#pragma unroll
        for (int i = 0; i < G; ++i) {
          acc[i][j] = fmaf(xv.x, wv[i].x, acc[i][j]);
          acc[i][j] = fmaf(xv.y, wv[i].y, acc[i][j]);
          acc[i][j] = fmaf(xv.z, wv[i].z, acc[i][j]);
          acc[i][j] = fmaf(xv.w, wv[i].w, acc[i][j]);
        }
      }
    }
    __syncwarp();  // the stage that is filled next was read one chunk ago
    if (c + STAGES - 1 < chunks) {
      copy_w(c + STAGES - 1);
      copy_x(c + STAGES - 1);
    }
    copies_commit();
    if (++in_piece == piece_chunks || c + 1 == chunks) {
      end_piece();
      in_piece = 0;
    }
  }
  copies_wait<0>();
}

// MT: the most tokens.  CLUSTER 4: block r of a cluster takes quarter r, its warp v piece 4 r + v.  CLUSTER 1: warp v takes
// quarter v.
template <int MT, int CLUSTER>
__global__ void __launch_bounds__(STREAM_WARPS * 32, 3)
gemm_f32_stream_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                       float* __restrict__ out, int M, int N, int K, int ldx, int ldw, int ldo, int accum) {
  extern __shared__ __align__(16) float smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ring = smem + warp * STREAM_STAGES<MT> * STREAM_STAGE<MT>;
  const int n0 = (int)(blockIdx.x / CLUSTER) * 32;
  x += (size_t)blockIdx.y * MT * ldx;
  out += (size_t)blockIdx.y * MT * ldo;
  M = min(MT, M - (int)blockIdx.y * MT);
  const int piece = piece_length(K);
  const int rank = CLUSTER > 1 ? (int)cluster_rank() : 0;
  const int span = CLUSTER > 1 ? piece : 4 * piece;
  const int k_begin = min(K, (CLUSTER > 1 ? 4 * rank + warp : warp) * span), k_end = min(K, k_begin + span);
  tl::pdl_launch_dependents();  // the next kernel may start its own prologue
  constexpr int G = TG<MT>;
  float acc[G][MT / G], sum[G][MT / G];
#pragma unroll
  for (int i = 0; i < G; ++i)
#pragma unroll
    for (int j = 0; j < MT / G; ++j) acc[i][j] = sum[i][j] = 0.f;
  stream_range<MT>(ring, x, w, M, N, K, ldx, ldw, n0, k_begin, k_end, piece, acc, [&]() {
#pragma unroll
    for (int i = 0; i < G; ++i)
#pragma unroll
      for (int j = 0; j < MT / G; ++j) {
        sum[i][j] += acc[i][j];
        acc[i][j] = 0.f;
      }
  });
  __syncthreads();  // the rings are free
  float* sums = smem;  // [4 warps][MT][32]
#pragma unroll
  for (int i = 0; i < G; ++i)
#pragma unroll
    for (int j = 0; j < MT / G; ++j) sums[(warp * MT + j * G + lane % G) * 32 + lane / G + i * (32 / G)] = sum[i][j];
  __syncthreads();
  if constexpr (CLUSTER == 1) {
    for (int m = warp; m < M; m += STREAM_WARPS)
      if (n0 + lane < N) {
        float v = 0.f;
#pragma unroll
        for (int s = 0; s < 4; ++s) v += sums[(s * MT + m) * 32 + lane];
        put(out + (size_t)m * ldo + n0 + lane, bias, accum, n0 + lane, v);
      }
  } else {
    float* quarter = smem + 4 * MT * 32;  // [MT][32]
    for (int m = warp; m < MT; m += STREAM_WARPS) {
      float v = 0.f;
#pragma unroll
      for (int s = 0; s < 4; ++s) v += sums[(s * MT + m) * 32 + lane];
      quarter[m * 32 + lane] = v;
    }
    cluster_sync();
    for (int m = 4 * warp + rank; m < M; m += 4 * STREAM_WARPS)
      if (n0 + lane < N) {
        float v = 0.f;
#pragma unroll
        for (int s = 0; s < 4; ++s) v += peer_read(quarter + m * 32 + lane, s);
        put(out + (size_t)m * ldo + n0 + lane, bias, accum, n0 + lane, v);
      }
    cluster_sync();  // nobody leaves while a peer may still read its memory
  }
}

// Two packed fused multiply-adds, each rounded like a single one.
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

constexpr int TILE_K = 16;
// TC: columns of a thread's tile of 8 rows
template <int TILE_M, int TILE_N, int TC> constexpr int TILE_THREADS = (TILE_M / 8) * (TILE_N / TC);
// two stages of both operands, k-major, and the tile's sums
template <int TILE_M, int TILE_N> constexpr int TILE_SMEM = 2 * TILE_K * (TILE_M + 4 + TILE_N + 4) * 4 + TILE_M * TILE_N * 4;

// A thread's outputs: rows 4 ty + {0..3} and TILE_M / 2 + 4 ty + {0..3}, columns 4 tx + {0..3} and (TC 8)
// TILE_N / 2 + 4 tx + {0..3}, so that a quarter warp's 16-byte reads lie side by side.
// BESIDE: the tiles from number ``whole`` on of a product whose others are the launch just before; else those below it.
template <int TILE_M, int TILE_N, int TC, int CLUSTER, bool BESIDE>
__global__ void __launch_bounds__(TILE_THREADS<TILE_M, TILE_N, TC>, (TC == 8 ? 256 : 512) / TILE_THREADS<TILE_M, TILE_N, TC>)
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                     float* __restrict__ out, int M, int N, int K, int ldx, int ldw, int ldo, int accum, int whole) {
  constexpr int NT = TILE_THREADS<TILE_M, TILE_N, TC>;
  constexpr int XS = TILE_M + 4, WS = TILE_N + 4;
  constexpr int STAGE = TILE_K * (XS + WS);
  constexpr int X4 = TILE_M * TILE_K / 4 / NT, W4 = TILE_N * TILE_K / 4 / NT;  // 16-byte reads a thread
  extern __shared__ __align__(16) float smem[];
  float* sums = smem + 2 * STAGE;  // [TILE_M][TILE_N]: the total so far, or this block's quarter
  const int tid = threadIdx.x;
  const int tx = tid % (TILE_N / TC), ty = tid / (TILE_N / TC);
  const int rank = CLUSTER > 1 ? (int)cluster_rank() : 0;
  int m0 = blockIdx.y * TILE_M, n0 = (int)(blockIdx.x / CLUSTER) * TILE_N;
  if constexpr (BESIDE) {
    const int tile = whole + (int)(blockIdx.x / CLUSTER), across = (N + TILE_N - 1) / TILE_N;
    m0 = tile / across * TILE_M;
    n0 = tile % across * TILE_N;
  } else if (CLUSTER == 1 && (int)(blockIdx.y * gridDim.x + blockIdx.x) >= whole) {
    return;  // another launch's tile
  }
  const int piece = piece_length(K);
  const int k_begin = CLUSTER > 1 ? min(K, rank * 4 * piece) : 0;
  const int k_end = CLUSTER > 1 ? min(K, k_begin + 4 * piece) : K;
  // Everything before us in the stream is complete and visible after the wait.  The launch just before a BESIDE one is the same
  // product's other tiles, of which this one reads nothing and every block of which has waited, or left, before this grid
  // could start; the wait moves to the end.
  if (!BESIDE) tl::pdl_wait();
  tl::pdl_launch_dependents();  // the next kernel may start its own prologue

  float4 xr[X4], wr[W4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < X4; ++i) {
      const int e = tid + i * NT, r = e / (TILE_K / 4), k = k0 + e % (TILE_K / 4) * 4;
      xr[i] = (m0 + r < M && k < k_end) ? *reinterpret_cast<const float4*>(x + (size_t)(m0 + r) * ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < W4; ++i) {
      const int e = tid + i * NT, r = e / (TILE_K / 4), k = k0 + e % (TILE_K / 4) * 4;
      wr[i] = (n0 + r < N && k < k_end) ? *reinterpret_cast<const float4*>(w + (size_t)(n0 + r) * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto stash = [&](float* stage) {
#pragma unroll
    for (int i = 0; i < X4; ++i) {
      const int e = tid + i * NT, r = e / (TILE_K / 4), k = e % (TILE_K / 4) * 4;
      stage[(k + 0) * XS + r] = xr[i].x;
      stage[(k + 1) * XS + r] = xr[i].y;
      stage[(k + 2) * XS + r] = xr[i].z;
      stage[(k + 3) * XS + r] = xr[i].w;
    }
    float* ws = stage + TILE_K * XS;
#pragma unroll
    for (int i = 0; i < W4; ++i) {
      const int e = tid + i * NT, r = e / (TILE_K / 4), k = e % (TILE_K / 4) * 4;
      ws[(k + 0) * WS + r] = wr[i].x;
      ws[(k + 1) * WS + r] = wr[i].y;
      ws[(k + 2) * WS + r] = wr[i].z;
      ws[(k + 3) * WS + r] = wr[i].w;
    }
  };
  unsigned long long acc[8][TC / 2], quarter[8][TC / 2];  // pairs of neighbouring columns
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TC / 2; ++j) acc[i][j] = quarter[i][j] = 0ull;
  auto row_of = [&](int i) { return (i < 4 ? 0 : TILE_M / 2) + 4 * ty + (i & 3); };
  auto col_of = [&](int j) { return (j < 2 ? 0 : TILE_N / 2) + 4 * tx + 2 * (j & 1); };
  // quarter += acc; at a quarter's end it goes into ``sums`` (first: it replaces what is there)
  auto end_piece = [&](bool quarter_ends, bool first) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TC / 2; ++j) {
        float2 q = unpack2(quarter[i][j]);
        const float2 a = unpack2(acc[i][j]);
        q.x += a.x;
        q.y += a.y;
        acc[i][j] = 0ull;
        if (quarter_ends) {
          float2* s = reinterpret_cast<float2*>(sums + row_of(i) * TILE_N + col_of(j));
          if (!first) {
            const float2 old = *s;
            q.x = old.x + q.x;
            q.y = old.y + q.y;
          }
          *s = q;
          q = make_float2(0.f, 0.f);
        }
        quarter[i][j] = pack2(q.x, q.y);
      }
  };

  const int steps = k_end > k_begin ? (k_end - k_begin + TILE_K - 1) / TILE_K : 0;
  const int piece_steps = piece / TILE_K;
  if (steps) {
    fetch(k_begin);
    stash(smem);
  }
  __syncthreads();
  int in_piece = 0, pieces = 0;
  bool first = true;
  for (int it = 0; it < steps; ++it) {
    const float* xs = smem + (it & 1) * STAGE;
    const float* ws = xs + TILE_K * XS;
    if (it + 1 < steps) fetch(k_begin + (it + 1) * TILE_K);
#pragma unroll
    for (int k = 0; k < TILE_K; ++k) {
      const float4 x0 = *reinterpret_cast<const float4*>(xs + k * XS + 4 * ty);
      const float4 x1 = *reinterpret_cast<const float4*>(xs + k * XS + TILE_M / 2 + 4 * ty);
      const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(ws + k * WS + 4 * tx);
      ulonglong2 w1;
      if constexpr (TC == 8) w1 = *reinterpret_cast<const ulonglong2*>(ws + k * WS + TILE_N / 2 + 4 * tx);
      const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned long long xx = pack2(xv[i], xv[i]);
        fma2(acc[i][0], xx, w0.x);
        fma2(acc[i][1], xx, w0.y);
        if constexpr (TC == 8) {
          fma2(acc[i][2], xx, w1.x);
          fma2(acc[i][3], xx, w1.y);
        }
      }
    }
    if (++in_piece == piece_steps || it + 1 == steps) {
      const bool ends = ++pieces == 4 || it + 1 == steps;
      end_piece(ends, first);
      if (ends) {
        first = false;
        pieces = 0;
      }
      in_piece = 0;
    }
    if (it + 1 < steps) stash(smem + ((it + 1) & 1) * STAGE);  // (read last one step ago, before the barrier)
    __syncthreads();
  }
  if (CLUSTER > 1 && first)  // a quarter past the end of K
    for (int e = tid; e < TILE_M * TILE_N; e += NT) sums[e] = 0.f;
  if (CLUSTER > 1) cluster_sync();
  else __syncthreads();
  for (int e = tid; e < TILE_M / CLUSTER * TILE_N; e += NT) {
    const int r = rank * (TILE_M / CLUSTER) + e / TILE_N, c = e % TILE_N;
    if (m0 + r >= M || n0 + c >= N) continue;
    float v;
    if constexpr (CLUSTER == 1) {
      v = sums[r * TILE_N + c];
    } else {
      v = 0.f;
#pragma unroll
      for (int s = 0; s < CLUSTER; ++s) v += peer_read(sums + r * TILE_N + c, s);
    }
    put(out + (size_t)(m0 + r) * ldo + n0 + c, bias, accum, n0 + c, v);
  }
  if (CLUSTER > 1) cluster_sync();  // nobody leaves while a peer may still read its memory
  if (BESIDE) tl::pdl_wait();
}

template <int CLUSTER, typename Kernel, typename... Args>
int launch_clusters(Kernel kernel, bool& configured, dim3 grid, int threads, int smem, cudaStream_t stream, Args... args) {
  if (!configured) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return (int)err;
    configured = true;
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = CLUSTER;
  attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = tl::pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&config, kernel, args...);
  return TL_LAUNCH_CHECK();
}

int sm_count() {
  static int sms = 0;
  if (sms <= 0) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
      sms = 148;
  }
  return sms;
}

// The kernel, its tile and its split follow from the sizes; the bits depend on none of them.  Every form was measured at K 4 to
// 4096, N 32 to 12288 and M 1 to 2048; the lines:
// - Four blocks a cluster where all of them are resident at once, or K is long enough to pay for a second wave, and not at all
//   where most quarters of K are empty (17 rows, K 4 x N 4096: 9.1 us as clusters, 2.4 in one block; 509 rows, 64 x 4096: 46 and 11;
//   2 rows, 512 x 4096: 6.0 and 3.6, 4096 x 4096: 18.6 and 22.5).
// - 17 to 32 rows, and up to 128 of narrow products: the stream kernel, 32 rows a block, has the shorter chains (64 rows, K x N
//   4864 x 896: 35 against 69 us; 896 x 1152: 11 against 17); on wider products the tiles read the weights less often (64 rows,
//   896 x 9728: 52 us against two passes of 26), on short K they start faster (17 rows, 32 x 2048: 2.8 us against 4.6).
// - Small tiles for up to 128 rows, and for short K until they take two waves (509 rows, 256 x 2048: 13 us, 21 with large ones).
constexpr int SHORT_K = 64, NARROW = 2048;

template <int MT>
int launch_stream(const float* x, const float* w, const float* bias, float* out, int accum, int M, int N, int K, int ldx,
                  int ldw, int ldo, cudaStream_t stream) {
  const int tiles = (N + 31) / 32, down = (M + MT - 1) / MT;
  static bool configured[2] = {false, false};
  const bool together = 4ll * tiles * down <= 3 * sm_count();
  if (K > SHORT_K && (together || (K >= (MT <= 16 ? 1024 : 512) && tiles < 2 * sm_count())))
    return launch_clusters<4>(gemm_f32_stream_kernel<MT, 4>, configured[1], dim3(4 * tiles, down), STREAM_WARPS * 32,
                              STREAM_SMEM<MT>, stream, x, w, bias, out, M, N, K, ldx, ldw, ldo, accum);
  return launch_clusters<1>(gemm_f32_stream_kernel<MT, 1>, configured[0], dim3(tiles, down), STREAM_WARPS * 32, STREAM_SMEM<MT>,
                            stream, x, w, bias, out, M, N, K, ldx, ldw, ldo, accum);
}

// Blocks of a tile size that are resident at once.
template <int TILE_M, int TILE_N, int TC> int resident() { return sm_count() * ((TC == 8 ? 256 : 512) / TILE_THREADS<TILE_M, TILE_N, TC>); }

template <int TILE_M, int TILE_N, int TC>
int launch_tiles(const float* x, const float* w, const float* bias, float* out, int accum, int M, int N, int K, int ldx,
                 int ldw, int ldo, cudaStream_t stream) {
  const int across = (N + TILE_N - 1) / TILE_N, down = (M + TILE_M - 1) / TILE_M;
  const long long blocks = (long long)across * down, room = resident<TILE_M, TILE_N, TC>();
  constexpr int NT = TILE_THREADS<TILE_M, TILE_N, TC>;
  static bool configured[3] = {false, false, false};
  if ((K > 160 && 4 * blocks <= room) || (K >= 512 && blocks < room))
    return launch_clusters<4>(gemm_f32_tile_kernel<TILE_M, TILE_N, TC, 4, false>, configured[1], dim3(4 * across, down), NT,
                              TILE_SMEM<TILE_M, TILE_N>, stream, x, w, bias, out, M, N, K, ldx, ldw, ldo, accum, (int)blocks);
  // A last wave that is nearly empty takes as long as a full one: its tiles go to four blocks each, which start beside the
  // blocks that are still at work.  (K x N 896 x 9728: 509 rows, 608 tiles for 296 blocks, 249 -> 212 us; 256 rows 159 -> 119;
  // 3584 x 3584, 700 rows: 614 -> 494.)
  const long long rest = blocks % room, whole = K >= 512 && blocks > room && 4 * rest <= room ? blocks - rest : blocks;
  const int rc = launch_clusters<1>(gemm_f32_tile_kernel<TILE_M, TILE_N, TC, 1, false>, configured[0], dim3(across, down), NT,
                                    TILE_SMEM<TILE_M, TILE_N>, stream, x, w, bias, out, M, N, K, ldx, ldw, ldo, accum, (int)whole);
  if (rc || whole == blocks) return rc;
  return launch_clusters<4>(gemm_f32_tile_kernel<TILE_M, TILE_N, TC, 4, true>, configured[2], dim3(4 * (unsigned)rest), NT,
                            TILE_SMEM<TILE_M, TILE_N>, stream, x, w, bias, out, M, N, K, ldx, ldw, ldo, accum, (int)whole);
}

int launch_f32(const float* x, const float* w, const float* bias, float* out, int accum, int M, int N, int K, int ldx,
               int ldw, int ldo, cudaStream_t stream) {
  if (M <= 1) return launch_stream<1>(x, w, bias, out, accum, M, N, K, ldx, ldw, ldo, stream);
  if (M <= 4) return launch_stream<4>(x, w, bias, out, accum, M, N, K, ldx, ldw, ldo, stream);
  if (M <= 8) return launch_stream<8>(x, w, bias, out, accum, M, N, K, ldx, ldw, ldo, stream);
  if (M <= 16) return launch_stream<16>(x, w, bias, out, accum, M, N, K, ldx, ldw, ldo, stream);
  if (K > SHORT_K && (M <= 32 || (M <= 128 && N <= NARROW)))
    return launch_stream<32>(x, w, bias, out, accum, M, N, K, ldx, ldw, ldo, stream);
  const long long small = (long long)((N + 63) / 64) * ((M + 63) / 64);
  if (K <= 512 ? small < 2 * resident<64, 64, 4>() : M <= 128)
    return launch_tiles<64, 64, 4>(x, w, bias, out, accum, M, N, K, ldx, ldw, ldo, stream);
  return launch_tiles<128, 64, 8>(x, w, bias, out, accum, M, N, K, ldx, ldw, ldo, stream);
}

template <typename T, typename OutT>
int launch(const void* x, const void* w, const float* bias, void* out, int accumulate, int M, int N,
           int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return TL_ERR_UNSUPPORTED;
  if (accumulate)
    tl::launch_kernel(gemm_simt_kernel<T, OutT, true>, grid, 256, 0, stream, (const T*)x, (const T*)w, bias, (OutT*)out, M, N, K, ldx, ldw, ldo);
  else
    tl::launch_kernel(gemm_simt_kernel<T, OutT, false>, grid, 256, 0, stream, (const T*)x, (const T*)w, bias, (OutT*)out, M, N, K, ldx, ldw, ldo);
  return TL_LAUNCH_CHECK();
}

}  // namespace

extern "C" int tl_gemm_simt(const void* x, const void* w, int in_dtype, const float* bias, void* out,
                            int out_dtype, int accumulate, int M, int N, int K, int ldx, int ldw,
                            int ldo, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return TL_ERR_UNSUPPORTED;
  if (in_dtype == TL_DTYPE_F32) {
    if (out_dtype != TL_DTYPE_F32) return TL_ERR_UNSUPPORTED;
    // 16-byte copies along K: rows and their ends on 16-byte boundaries
    const bool wide = K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 &&
                      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    if (wide && (M + 127) / 128 <= 65535)
      return launch_f32((const float*)x, (const float*)w, bias, (float*)out, accumulate, M, N, K, ldx, ldw, ldo, stream);
    return launch<float, float>(x, w, bias, out, accumulate, M, N, K, ldx, ldw, ldo, stream);
  }
  if (out_dtype == TL_DTYPE_F32)
    return launch<__nv_bfloat16, float>(x, w, bias, out, accumulate, M, N, K, ldx, ldw, ldo, stream);
  return launch<__nv_bfloat16, __nv_bfloat16>(x, w, bias, out, accumulate, M, N, K, ldx, ldw, ldo, stream);
}
