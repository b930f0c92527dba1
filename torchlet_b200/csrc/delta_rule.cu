// The generalized delta rule: a recurrent mixer whose per-request state is one D x D
// float32 matrix per head (key channel i, value channel j), carried from token to token:
//
//   S_t = diag(w_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T,    o_t = S_t^T r_t
//
// with u = k / sqrt(sum(k^2) + 1e-6), decay w = exp(-exp(-1/2) sigmoid(W2 tanh(l) + w0)) in
// (0.545, 1) and removal rate a = sigmoid(a' + b).  Everything here is float32, also in the
// bfloat16 engine: the projections arrive as float32 rows
//   proj[t] = [ r (H D) | k (H D) | v (H D) | g (H D) | a' (H D) | l (rank) ].
//
// Three kernels:
//   prepare  one block per (8 tokens, head), or (token, head) where few: w, u and a * u of every key channel;
//   scan     one block per (request, head) or 16 columns of one: the columns of S are independent of one another;
//            four lanes share a column, each keeps a quarter of it in registers (and serves two
//            columns, so that the vectors it reads are used twice), and the block
//            walks the request's tokens of this step in order; r, k, v, w, u, a*u of a few tokens
//            at a time are staged in shared memory (two stages, asynchronous copies).  The state
//            row of the request's slot is read at the start and written back at the end, so a
//            prompt cut into portions, or decoded token by token, runs the same additions in the
//            same order as the whole prompt;
//   finish   one warp per (token, head): o / rms(o) * weight * sigmoid(g) in the compute type.
#include <math.h>

#include "common.cuh"

namespace {

using namespace tl;

constexpr float DECAY_RATE = 0.6065306597126334f;  // exp(-1/2)

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }

// Tokens a block of the prepare kernel takes: eight, so that a W2 entry is read once for all, or one where the grid of eights
// would leave most SMs idle (8 tokens, 32 heads of 64, in a decode step: 20.4 -> 6.8 us; the bits
// are the same).
constexpr int PREP_TOKENS = 8;

// w2t: W2 transposed, [rank, heads * dim], so that the threads of a block read consecutive entries.
template <int NT, int TOKENS>
__global__ void __launch_bounds__(NT)
delta_prepare_kernel(const float* __restrict__ proj, int proj_stride, const float* __restrict__ w2t,
                     const float* __restrict__ w0, const float* __restrict__ a_bias, float* __restrict__ gates,
                     int tokens, int heads, int dim, int rank) {
  tl::pdl_launch_dependents();
  tl::pdl_wait();
  extern __shared__ float lowrank[];  // tanh(l): TOKENS x rank floats
  __shared__ float scratch[TOKENS][32];
  const int t0 = blockIdx.x * TOKENS, h = blockIdx.y, i = threadIdx.x;
  const int count = tokens - t0 < TOKENS ? tokens - t0 : TOKENS;
  const int hd = heads * dim;
  for (int e = threadIdx.x; e < TOKENS * rank; e += NT) {
    const int tt = e / rank, j = e - tt * rank;
    lowrank[e] = tt < count ? tanhf(proj[(size_t)(t0 + tt) * proj_stride + 5 * hd + j]) : 0.f;
  }
  __syncthreads();
  const bool on = i < dim;
  const int c = h * dim + (on ? i : 0);
  float inner[TOKENS];
#pragma unroll
  for (int tt = 0; tt < TOKENS; ++tt) inner[tt] = w0[c];
  if (on) {
#pragma unroll(TOKENS == 1 ? 32 : 8)
    for (int j = 0; j < rank; ++j) {
      const float w = w2t[(size_t)j * hd + c];
#pragma unroll
      for (int tt = 0; tt < TOKENS; ++tt) inner[tt] = fmaf(w, lowrank[tt * rank + j], inner[tt]);
    }
  }
  // the tokens' keys are read and their squares summed together (the additions of block_sum, one barrier for all): a token after
  // the other the kernel waited eight times for a read and two barriers.  2,048 tokens, 32 heads of 64: 80 us against 90.
  float k[TOKENS], ss[TOKENS];
#pragma unroll
  for (int tt = 0; tt < TOKENS; ++tt) k[tt] = on && tt < count ? proj[(size_t)(t0 + tt) * proj_stride + hd + c] : 0.f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int tt = 0; tt < TOKENS; ++tt) {
    ss[tt] = warp_sum(k[tt] * k[tt]);
    if (lane == 0) scratch[tt][warp] = ss[tt];
  }
  __syncthreads();
#pragma unroll
  for (int tt = 0; tt < TOKENS; ++tt) ss[tt] = warp_sum(lane < NT / 32 ? scratch[tt][lane] : 0.f);
  if (!on) return;
#pragma unroll
  for (int tt = 0; tt < TOKENS; ++tt) {
    if (tt >= count) break;  // (the same for every thread of the block)
    const float w = expf(-DECAY_RATE * sigmoidf_(inner[tt]));
    const float a = sigmoidf_(proj[(size_t)(t0 + tt) * proj_stride + 4 * hd + c] + a_bias[c]);
    const float u = k[tt] / sqrtf(ss[tt] + 1e-6f);
    float* out = gates + ((size_t)(t0 + tt) * heads + h) * 3 * dim;
    out[i] = w;
    out[dim + i] = u;
    out[2 * dim + i] = a * u;
  }
}

__device__ __forceinline__ void copy16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One block per (request, head).  Four lanes share a column of S (value channel j): lane part p
// keeps the key channels i with (i / 4) % 4 == p, and the two sums over i of a token (u^T S and
// S^T r) meet by two shuffles.  A lane serves CPL = 2 columns (j and j + D/2) with the same vector
// entries, so that what it reads from shared memory is used twice: with many blocks the kernel is bound by the
// shared-memory wavefronts of these reads.  All warps of the block read the same staged r, k, v,
// w, u, a*u of CHUNK tokens, two stages deep: while the block walks one chunk, the next is on its
// way (16-byte asynchronous copies where D and the row stride are multiples of 4 floats, plain
// loads otherwise).
//
// Few (request, head) pairs leave SMs idle and a block then waits for its own chain (read, four sums, shuffles, update): COLS 16 lets
// DK / 16 blocks take 16 columns of a head each, one column a lane, with a chunk's tokens unrolled so that the next token's
// reads pass the chain of this one.  The sums of a column, and so its bits, are the same.  One request of 2,048 tokens at 32
// heads of 64: 342 us against 812.
constexpr int KS = 4;
constexpr int SPLIT_COLS = 16;
__host__ __device__ constexpr int scan_chunk(int dk) { return dk <= 64 ? 8 : (dk <= 128 ? 4 : 2); }

template <int DK, bool VEC, int COLS, bool LONG>
__global__ void __launch_bounds__(COLS * KS / (COLS == DK ? 2 : 1))
delta_scan_kernel(const float* __restrict__ proj, int proj_stride, const float* __restrict__ gates,
                  const int* __restrict__ req_indptr, const int* __restrict__ slots, float* __restrict__ state,
                  float* __restrict__ out, int heads, int dim, int below, int max_slots) {
  tl::pdl_launch_dependents();
  tl::pdl_wait();
  constexpr int CPL = COLS == DK ? 2 : 1;  // columns a lane serves
  constexpr int NT = COLS * KS / CPL;
  constexpr int PER = DK / KS;  // key channels a lane keeps of each of its columns
  constexpr int CHUNK = scan_chunk(DK);
  __shared__ __align__(16) float stage[2][CHUNK][6][DK];  // r, k, v, w, u, a*u
  const int req = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int part = tid % KS;
  int col[CPL];
  bool on[CPL];
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    col[c] = blockIdx.z * COLS + tid / KS + c * (COLS / CPL);
    on[c] = col[c] < dim;
  }
  const int hd = heads * dim;
  const int first = req_indptr[req], last = req_indptr[req + 1];
  if (last - first >= below) return;  // its tokens are another kernel's
  const int slot = slots[req];
  const bool live = TL_DEBUG_OK(slot >= -1 && slot < max_slots, TL_DEBUG_SLOT, slot) && slot >= 0;
  if (!live) {  // a padding lane of a captured step: no state is touched
    if (part == 0)
      for (int t = first; t < last; ++t)
#pragma unroll
        for (int c = 0; c < CPL; ++c)
          if (on[c]) out[(size_t)t * hd + h * dim + col[c]] = 0.f;
    return;
  }
  if (!VEC || dim < DK) {  // entries past dim stay zero in both stages
    for (int e = tid; e < 2 * CHUNK * 6 * DK; e += NT) (&stage[0][0][0][0])[e] = 0.f;
    __syncthreads();
  }
  // 16-byte copies: a thread's entries of a chunk are the same in every chunk, so for whole chunks (LONG) their sources are worked
  // out once and move on by a chunk (with the divisions in the loop a block of 64 threads spent more on them than on the
  // recurrence); for a token or a few, whose kernel is as long as its start, that is the longer way (32 heads of 64, one
  // token: 2.8 us against 2.3)
  constexpr int QUADS = DK / 4, COPIES = (CHUNK * 6 * QUADS + NT - 1) / NT;
  const float* source[LONG ? COPIES : 1];
  if constexpr (LONG) {
#pragma unroll
    for (int i = 0; i < COPIES; ++i) {
      const int e = tid + i * NT, tt = e / (6 * QUADS), what = e / QUADS % 6, q = e % QUADS;
      const size_t t = (size_t)first + tt;
      source[i] = what < 3 ? proj + t * proj_stride + what * hd + h * dim + 4 * q
                           : gates + ((t * heads + h) * 3 + (what - 3)) * dim + 4 * q;
    }
  }
  auto fetch = [&](int base, int buf) {
    const int count = last - base < CHUNK ? last - base : CHUNK;
    if constexpr (LONG) {
      const int quads = dim >> 2;
#pragma unroll
      for (int i = 0; i < COPIES; ++i) {
        const int e = tid + i * NT, tt = e / (6 * QUADS), what = e / QUADS % 6, q = e % QUADS;
        if (tt < count && q < quads) copy16(&stage[buf][tt][what][4 * q], source[i]);
        source[i] += (size_t)CHUNK * (what < 3 ? proj_stride : heads * 3 * dim);
      }
    } else if constexpr (VEC) {
      const int quads = dim >> 2;
      for (int e = tid; e < count * 6 * quads; e += NT) {
        const int tt = e / (6 * quads), rest = e - tt * 6 * quads, what = rest / quads, q = rest - what * quads;
        const int t = base + tt;
        const float* src = what < 3 ? proj + (size_t)t * proj_stride + what * hd + h * dim
                                    : gates + (((size_t)t * heads + h) * 3 + (what - 3)) * dim;
        copy16(&stage[buf][tt][what][4 * q], src + 4 * q);
      }
    } else {
      for (int e = tid; e < count * 6 * dim; e += NT) {
        const int tt = e / (6 * dim), rest = e - tt * 6 * dim, what = rest / dim, i = rest - what * dim;
        const int t = base + tt;
        stage[buf][tt][what][i] = what < 3 ? proj[(size_t)t * proj_stride + what * hd + h * dim + i]
                                           : gates[(((size_t)t * heads + h) * 3 + (what - 3)) * dim + i];
      }
    }
    copies_commit();
  };
  if (first < last) fetch(first, 0);

  // this lane's key channels: i = 4 (q KS + part) + e, q = 0 .. PER/4 - 1, e = 0 .. 3
  float* mine = state + ((size_t)slot * heads + h) * dim * dim;
  float S[CPL][PER];
#pragma unroll
  for (int c = 0; c < CPL; ++c)
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      const int i = 4 * ((n >> 2) * KS + part) + (n & 3);
      S[c][n] = (on[c] && i < dim) ? mine[(size_t)i * dim + col[c]] : 0.f;
    }

  int buf = 0;
  for (int base = first; base < last; base += CHUNK, buf ^= 1) {
    const int count = last - base < CHUNK ? last - base : CHUNK;
    if (base + CHUNK < last) {
      fetch(base + CHUNK, buf ^ 1);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
    auto token = [&](const int tt) {
      const int t = base + tt;
      const float4* r4 = reinterpret_cast<const float4*>(stage[buf][tt][0]);
      const float4* k4 = reinterpret_cast<const float4*>(stage[buf][tt][1]);
      const float4* w4 = reinterpret_cast<const float4*>(stage[buf][tt][3]);
      const float4* u4 = reinterpret_cast<const float4*>(stage[buf][tt][4]);
      const float4* au4 = reinterpret_cast<const float4*>(stage[buf][tt][5]);
      float v[CPL], seen[CPL], o[CPL];
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        v[c] = stage[buf][tt][2][col[c] & (DK - 1)];
        seen[c] = 0.f;
        o[c] = 0.f;
      }
      float part_seen[CPL][4];
#pragma unroll
      for (int c = 0; c < CPL; ++c) part_seen[c][0] = part_seen[c][1] = part_seen[c][2] = part_seen[c][3] = 0.f;
#pragma unroll
      for (int q = 0; q < PER / 4; ++q) {
        const float4 u = u4[q * KS + part];
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          part_seen[c][0] = fmaf(u.x, S[c][4 * q], part_seen[c][0]);
          part_seen[c][1] = fmaf(u.y, S[c][4 * q + 1], part_seen[c][1]);
          part_seen[c][2] = fmaf(u.z, S[c][4 * q + 2], part_seen[c][2]);
          part_seen[c][3] = fmaf(u.w, S[c][4 * q + 3], part_seen[c][3]);
        }
      }
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        seen[c] = (part_seen[c][0] + part_seen[c][1]) + (part_seen[c][2] + part_seen[c][3]);
        seen[c] += __shfl_xor_sync(0xffffffffu, seen[c], 1);
        seen[c] += __shfl_xor_sync(0xffffffffu, seen[c], 2);
      }
      float part_o[CPL][4];
#pragma unroll
      for (int c = 0; c < CPL; ++c) part_o[c][0] = part_o[c][1] = part_o[c][2] = part_o[c][3] = 0.f;
#pragma unroll
      for (int q = 0; q < PER / 4; ++q) {
        const float4 w = w4[q * KS + part], au = au4[q * KS + part], k = k4[q * KS + part], r = r4[q * KS + part];
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          S[c][4 * q] = fmaf(k.x, v[c], fmaf(-au.x, seen[c], w.x * S[c][4 * q]));
          S[c][4 * q + 1] = fmaf(k.y, v[c], fmaf(-au.y, seen[c], w.y * S[c][4 * q + 1]));
          S[c][4 * q + 2] = fmaf(k.z, v[c], fmaf(-au.z, seen[c], w.z * S[c][4 * q + 2]));
          S[c][4 * q + 3] = fmaf(k.w, v[c], fmaf(-au.w, seen[c], w.w * S[c][4 * q + 3]));
          part_o[c][0] = fmaf(r.x, S[c][4 * q], part_o[c][0]);
          part_o[c][1] = fmaf(r.y, S[c][4 * q + 1], part_o[c][1]);
          part_o[c][2] = fmaf(r.z, S[c][4 * q + 2], part_o[c][2]);
          part_o[c][3] = fmaf(r.w, S[c][4 * q + 3], part_o[c][3]);
        }
      }
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        o[c] = (part_o[c][0] + part_o[c][1]) + (part_o[c][2] + part_o[c][3]);
        o[c] += __shfl_xor_sync(0xffffffffu, o[c], 1);
        o[c] += __shfl_xor_sync(0xffffffffu, o[c], 2);
        if (on[c] && part == 0) out[(size_t)t * hd + h * dim + col[c]] = o[c];
      }
    };
    if (COLS < DK && count == CHUNK) {
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) token(tt);
    } else {
#pragma unroll 1
      for (int tt = 0; tt < count; ++tt) token(tt);
    }
    __syncthreads();  // the stage is free for the chunk after the next
  }
#pragma unroll
  for (int c = 0; c < CPL; ++c)
    if (on[c]) {
#pragma unroll
      for (int n = 0; n < PER; ++n) {
        const int i = 4 * ((n >> 2) * KS + part) + (n & 3);
        if (i < dim) mine[(size_t)i * dim + col[c]] = S[c][n];
      }
    }
}

constexpr int FINISH_WARPS = 4;

template <typename T>
__global__ void __launch_bounds__(FINISH_WARPS * 32)
delta_finish_kernel(const float* __restrict__ o, const float* __restrict__ proj, int proj_stride,
                    const float* __restrict__ weight, T* __restrict__ out, long long items, int heads, int dim,
                    float eps) {
  tl::pdl_launch_dependents();
  tl::pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * FINISH_WARPS + warp;
  if (item >= items) return;
  const long long t = item / heads;
  const int h = (int)(item % heads);
  const int hd = heads * dim;
  const float* row = o + (size_t)t * hd + h * dim;
  float ss = 0.f;
  for (int i = lane; i < dim; i += 32) ss = fmaf(row[i], row[i], ss);
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / (float)dim + eps);
  const float* gate = proj + (size_t)t * proj_stride + 3 * hd + h * dim;
  for (int i = lane; i < dim; i += 32)
    out[(size_t)t * hd + h * dim + i] = from_float<T>(row[i] * inv * weight[h * dim + i] * sigmoidf_(gate[i]));
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

// Whether a head's columns go to several blocks (the bits are the same).  Measured at head sizes 36 to 256, 1 to 384 (request,
// head) pairs and 1 to 512 tokens a request:
// - up to 64: a block of 16 columns is faster (128 tokens: 40 -> 25 us) only where at most two lie
//   on an SM (64 pairs of 64: 40 -> 34; 80 pairs: 40 -> 51), and its longer start has to be won back (64 pairs: 1 token 3.1 -> 4.2 us,
//   16 tokens 6.7 -> 10; 16 pairs: 16 tokens 6.5 -> 5.3);
// - up to 128: where at most four lie on an SM (64 pairs of 128: 1 token 5.3 -> 4.2 us, 128 tokens 111 -> 100; 80 pairs:
//   5.7 -> 6.3 and 112 -> 196);
// - beyond: the block of all columns is the slower one everywhere (148 pairs of 256: 1 token 48 -> 22 us, 512 tokens equal).
bool split_columns(int requests, int heads, int dim, int tokens) {
  const long long pairs = (long long)requests * heads, blocks = pairs * ((dim + SPLIT_COLS - 1) / SPLIT_COLS);
  if (dim <= 32) return false;
  if (dim <= 64) return blocks <= 2 * sm_count() && tokens >= (blocks <= sm_count() ? 16ll : 64ll) * requests;
  if (dim <= 128) return blocks <= 4 * sm_count();
  return pairs <= sm_count();
}

}  // namespace

TL_DEBUG_READER(tl_delta_rule_debug_error)

extern "C" {

// gates: float32 [tokens, heads, 3, dim] scratch;  w2t: [rank, heads * dim].
int tl_delta_prepare(const float* proj, int proj_stride, const float* w2t, const float* w0, const float* a_bias,
                     float* gates, int tokens, int heads, int dim, int rank, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (dim <= 0 || dim > 1024 || heads > 65535 || rank <= 0 || rank > 1024) return TL_ERR_UNSUPPORTED;
  const bool singly = (long long)((tokens + PREP_TOKENS - 1) / PREP_TOKENS) * heads <= sm_count();
  const int each = singly ? 1 : PREP_TOKENS;
  dim3 grid((tokens + each - 1) / each, heads);
  const size_t smem = (size_t)each * rank * sizeof(float);
#define TL_PREPARE_TOKENS(NT, TOKENS)                                                                                      \
  tl::launch_kernel(delta_prepare_kernel<NT, TOKENS>, grid, NT, smem, stream, proj, proj_stride, w2t, w0, a_bias, gates,   \
                    tokens, heads, dim, rank)
#define TL_PREPARE(NT)                            \
  if (singly) TL_PREPARE_TOKENS(NT, 1);           \
  else TL_PREPARE_TOKENS(NT, PREP_TOKENS)
  if (dim <= 32) { TL_PREPARE(32); }
  else if (dim <= 64) { TL_PREPARE(64); }
  else if (dim <= 128) { TL_PREPARE(128); }
  else if (dim <= 256) { TL_PREPARE(256); }
  else { TL_PREPARE(1024); }
#undef TL_PREPARE
#undef TL_PREPARE_TOKENS
  return TL_LAUNCH_CHECK();
}

// state: float32 [max_slots, heads, dim, dim]; out: float32 [tokens, heads * dim]; tokens: of all requests;
// requests of ``below`` tokens and more are left out (delta_chunked.cu).
int tl_delta_scan(const float* proj, int proj_stride, const float* gates, const int* req_indptr, const int* slots,
                  float* state, float* out, int requests, int heads, int dim, int tokens, int below,
                  int max_slots, cudaStream_t stream) {
  if (requests <= 0) return 0;
  if (dim <= 0 || dim > 256 || heads > 65535) return TL_ERR_UNSUPPORTED;
  dim3 grid(requests, heads);
  const bool vec = dim % 4 == 0 && proj_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(proj) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(gates) & 15) == 0;
  const bool split = split_columns(requests, heads, dim, tokens);
  // (head sizes up to 64: a chunk of 8 tokens; up to 128: 4 tokens 8.2 -> 7.6 us, 2 equal; beyond: 1 token 20 us against 22)
  // the blocks walk long enough that their places matter more than the larger shared memory's carve-out
  const bool long_walk = tokens >= 64ll * requests;
  const bool long_portions = vec && (dim > 128 || tokens >= (dim > 64 ? 4ll : 8ll) * requests);
#define TL_SCAN_INSTANCE(DK, VEC, COLS, LONG)                                                                       \
  tl::launch_apart<delta_scan_kernel<DK, VEC, COLS, LONG>>(grid, COLS * KS / (COLS == DK ? 2 : 1), long_walk, sm_count(), \
                                                          sizeof(float) * 2 * scan_chunk(DK) * 6 * DK, 0, stream, proj,  \
                                                          proj_stride, gates, req_indptr, slots, state, out, heads, dim, \
                                                          below, max_slots)
#define TL_SCAN_COLS(DK, COLS)                          \
  if (long_portions) TL_SCAN_INSTANCE(DK, true, COLS, true);    \
  else if (vec) TL_SCAN_INSTANCE(DK, true, COLS, (DK > 128)); \
  else TL_SCAN_INSTANCE(DK, false, COLS, false)
#define TL_SCAN(DK)                                     \
  if (split) {                                          \
    grid.z = (dim + SPLIT_COLS - 1) / SPLIT_COLS;       \
    TL_SCAN_COLS(DK, SPLIT_COLS);                       \
  } else {                                              \
    TL_SCAN_COLS(DK, DK);                               \
  }
  if (dim <= 16) { TL_SCAN_COLS(16, 16); }
  else if (dim <= 32) { TL_SCAN_COLS(32, 32); }
  else if (dim <= 64) { TL_SCAN(64); }
  else if (dim <= 128) { TL_SCAN(128); }
  else { TL_SCAN(256); }
#undef TL_SCAN
#undef TL_SCAN_COLS
#undef TL_SCAN_INSTANCE
  return TL_LAUNCH_CHECK();
}

int tl_delta_finish(const float* o, const float* proj, int proj_stride, const float* weight, void* out, int out_dtype,
                    int tokens, int heads, int dim, float eps, cudaStream_t stream) {
  const long long items = (long long)tokens * heads;
  if (items <= 0) return 0;
  const unsigned blocks = (unsigned)((items + FINISH_WARPS - 1) / FINISH_WARPS);
  if (out_dtype == TL_DTYPE_F32)
    tl::launch_kernel(delta_finish_kernel<float>, blocks, FINISH_WARPS * 32, 0, stream, o, proj, proj_stride, weight,
                      (float*)out, items, heads, dim, eps);
  else
    tl::launch_kernel(delta_finish_kernel<__nv_bfloat16>, blocks, FINISH_WARPS * 32, 0, stream, o, proj, proj_stride,
                      weight, (__nv_bfloat16*)out, items, heads, dim, eps);
  return TL_LAUNCH_CHECK();
}

}  // extern "C"
