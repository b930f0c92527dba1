// The generalized delta rule over long portions, a chunk of CHUNK tokens at a time: the numbers of delta_rule.cu's scan
//
//   y_t = S_(t-1)^T u_t,   S_t = diag(w_t) S_(t-1) - b_t y_t^T + k_t v_t^T,   o_t = S_t^T r_t,   b = a * u
//
// whose chain of dependent steps is a chunk long instead of a token.  With S the state at a chunk's start, P(s, t) the
// product of the decays w_(s+1) .. w_t per channel, and unrolled over the chunk:
//
//   y_t = S^T (u_t P(0, t-1)) + sum_(s < t)  MK[t][s] v_s - MB[t][s] y_s,   MK[t][s] = u_t . (P(s, t-1) k_s),  MB with b_s
//   o_t = S^T (r_t P(0, t))   + sum_(s <= t) NK[t][s] v_s - NB[t][s] y_s,   NK[t][s] = r_t . (P(s, t) k_s),    NB with b_s
//   S'  = diag(P(0, L)) S + sum_s (P(s, L) k_s) v_s^T - (P(s, L) b_s) y_s^T.
//
// The small triangular system for y does not know S: solved once, y_t = S^T W_t + X_t and o_t = S^T R_t + Z_t with
//
//   W_t = u_t P(0, t-1) - sum_(s < t)  MB[t][s] W_s,      X_t = sum_(s < t)  MK[t][s] v_s - MB[t][s] X_s,
//   R_t = r_t P(0, t)   - sum_(s <= t) NB[t][s] W_s,      Z_t = sum_(s <= t) NK[t][s] v_s - NB[t][s] X_s.
//
// Two kernels.  ``prepare`` (a block a (chunk, head), a thread a channel, all chunks at once; in place of the token-wise
// delta_prepare) computes the gates and these vectors; ``scan`` (a block a (request, head, 16 columns of S)) walks the
// chunks: 2 CHUNK sums over S that do not wait for one another, then one update of S.  Everything is float32; every decay
// between two tokens is a product of the decays between them, never a quotient.
//
// Error against 64 bits, whose sums differ in their order alone: 1.18e-7 against the scan's 1.13e-7 (random rows), 5.0 against
// 4.3e-7 (64 nearly equal keys, slow decays), 2.4 against 2.7e-6 (512 of them).
// One request of 2,048 tokens, 32 heads of 64: prepare 106 and scan 177 us against 80 and 362 token by token (0.69 us a chunk
// of 8; a chunk's reads one after the other instead of all ahead of their use: 1.1).  The
// order of a token's additions depends on where its chunk starts, so this form serves the bfloat16 engine; the float32
// engine, whose logits do not depend on how a sequence is cut, keeps the token-wise kernels.
#include <math.h>

#include "common.cuh"

namespace {

using namespace tl;

constexpr float DECAY_RATE = 0.6065306597126334f;  // exp(-1/2)
constexpr int CHUNK = 8, DK = 64, COLS = 16, GROUPS = DK / COLS;

// What prepare leaves of a (chunk, head), in floats:
//   P(0, L) [DK], then [token][W, R, P(s, L) k, P(s, L) b][DK], then for each group of COLS columns
//   [token][pair of columns][v, v, X, X] and [token][COLS] of Z.
constexpr int VECTORS = DK, COLUMNS = VECTORS + CHUNK * 4 * DK;
constexpr int GROUP = CHUNK * COLS / 2 * 4 + CHUNK * COLS, RECORD = COLUMNS + GROUPS * GROUP;

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }

// Requests of ``least`` tokens and more are cut into chunks; the others have none here.  A launch takes chunks [lo, hi) of each,
// in the order of the requests.
struct Pass {
  const int* req_indptr;
  int requests, least, lo, hi;
  __device__ __forceinline__ int chunks_of(int req) const {
    const int n = req < requests ? req_indptr[req + 1] - req_indptr[req] : 0;
    return n >= least ? max(0, min((n + CHUNK - 1) / CHUNK, hi) - lo) : 0;
  }
};

// Sums the 64 values of every lane over the warp: lane l is left with values 2 l and 2 l + 1, in v[0] and v[1].
__device__ __forceinline__ void scatter_sums(float (&v)[64], int lane) {
#pragma unroll
  for (int o = 16, n = 32; o > 0; o >>= 1, n >>= 1)
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const bool up = lane & o;
      const float send = up ? v[j] : v[j + n];
      v[j] = (up ? v[j + n] : v[j]) + __shfl_xor_sync(0xffffffffu, send, o);
    }
}
__host__ __device__ constexpr int below(int t, int s) { return t * (t - 1) / 2 + s; }         // s < t: 28 pairs
__host__ __device__ constexpr int upto(int t, int s) { return 28 + t * (t + 1) / 2 + s; }     // s <= t: 36 more

__global__ void __launch_bounds__(DK)
delta_chunk_prepare_kernel(const float* __restrict__ proj, int proj_stride, const float* __restrict__ w2t,
                           const float* __restrict__ w0, const float* __restrict__ a_bias, const Pass pass,
                           float* __restrict__ records, int heads, int dim, int rank) {
  tl::pdl_launch_dependents();
  extern __shared__ __align__(16) float lowrank[];  // tanh(l): [rank][CHUNK]
  __shared__ float squares[2][CHUNK];
  __shared__ float partial[2][2][64];  // [k, b][warp]: the pairs' sums over 32 channels
  __shared__ float pair[2][64];        // [k: MK, NK; b: MB, NB]
  const int h = blockIdx.y, i = threadIdx.x, lane = i & 31, warp = i >> 5;
  const int hd = heads * dim;
  // the request and the tokens of this chunk (every warp by itself)
  int id = blockIdx.x, first = -1, count = 0;
  for (int base = 0; base < pass.requests; base += 32) {
    const int mine = pass.chunks_of(base + lane);
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int before = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += before;
    }
    const unsigned beyond = __ballot_sync(0xffffffffu, sum > id);
    if (beyond) {
      const int at = __ffs(beyond) - 1;
      first = pass.req_indptr[base + at] + (pass.lo + id - __shfl_sync(0xffffffffu, sum - mine, at)) * CHUNK;
      count = min(CHUNK, pass.req_indptr[base + at + 1] - first);
      break;
    }
    id -= __shfl_sync(0xffffffffu, sum, 31);
  }
  tl::pdl_wait();
  if (first < 0) return;
  const float* rows = proj + (size_t)first * proj_stride;
  for (int e = i; e < CHUNK * rank; e += DK) {
    const int t = e / rank, j = e - t * rank;
    lowrank[j * CHUNK + t] = t < count ? tanhf(rows[(size_t)t * proj_stride + 5 * hd + j]) : 0.f;
  }
  const bool on = i < dim;
  const int c = h * dim + (on ? i : 0);
  float r[CHUNK], k[CHUNK], v[CHUNK], a[CHUNK];  // zero past the chunk's tokens and past dim
#pragma unroll
  for (int t = 0; t < CHUNK; ++t) {
    const float* row = rows + (size_t)t * proj_stride + c;
    const bool here = on && t < count;
    r[t] = here ? row[0] : 0.f;
    k[t] = here ? row[hd] : 0.f;
    v[t] = here ? row[2 * hd] : 0.f;
    a[t] = here ? row[4 * hd] : 0.f;
  }
  __syncthreads();
  float w[CHUNK];
#pragma unroll
  for (int t = 0; t < CHUNK; ++t) w[t] = w0[c];
#pragma unroll 8
  for (int j = 0; j < rank; ++j) {
    const float m = w2t[(size_t)j * hd + c];
    const float4 x = *reinterpret_cast<const float4*>(lowrank + j * CHUNK), y = *reinterpret_cast<const float4*>(lowrank + j * CHUNK + 4);
    const float l[CHUNK] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
    for (int t = 0; t < CHUNK; ++t) w[t] = fmaf(m, l[t], w[t]);
  }
#pragma unroll
  for (int t = 0; t < CHUNK; ++t) {
    const float ss = warp_sum(k[t] * k[t]);
    if (lane == 0) squares[warp][t] = ss;
  }
  __syncthreads();
  float u[CHUNK], b[CHUNK];
  const float bias = a_bias[c];
#pragma unroll
  for (int t = 0; t < CHUNK; ++t) {
    w[t] = on && t < count ? expf(-DECAY_RATE * sigmoidf_(w[t])) : 1.f;
    u[t] = k[t] / sqrtf((squares[0][t] + squares[1][t]) + 1e-6f);
    b[t] = sigmoidf_(a[t] + bias) * u[t];
  }
  float* record = records + ((size_t)blockIdx.x * heads + h) * RECORD;
  // this channel's share of the pairs' sums, first with k, then with b; what is left of k_s (b_s) at the chunk's end
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float sums[64];
#pragma unroll
    for (int s = 0; s < CHUNK; ++s) {
      float g = half ? b[s] : k[s];
      sums[upto(s, s)] = r[s] * g;
#pragma unroll
      for (int t = s + 1; t < CHUNK; ++t) {
        sums[below(t, s)] = u[t] * g;
        g *= w[t];
        sums[upto(t, s)] = r[t] * g;
      }
      record[VECTORS + (s * 4 + 2 + half) * DK + i] = g;
    }
    scatter_sums(sums, lane);
    partial[half][warp][2 * lane] = sums[0];
    partial[half][warp][2 * lane + 1] = sums[1];
  }
  __syncthreads();
  pair[0][i] = partial[0][0][i] + partial[0][1][i];
  pair[1][i] = partial[1][0][i] + partial[1][1][i];
  __syncthreads();
  float run = 1.f, W[CHUNK], X[CHUNK];
  float* columns = record + COLUMNS + (i / COLS) * GROUP;
  const int in_group = i % COLS;
#pragma unroll
  for (int t = 0; t < CHUNK; ++t) {
    float wt = u[t] * run, xt = 0.f;
    run *= w[t];
    float rt = r[t] * run, zt = 0.f;
#pragma unroll
    for (int s = 0; s < t; ++s) {
      const float mk = pair[0][below(t, s)], mb = pair[1][below(t, s)];
      wt = fmaf(-mb, W[s], wt);
      xt = fmaf(mk, v[s], fmaf(-mb, X[s], xt));
    }
    W[t] = wt;
    X[t] = xt;
#pragma unroll
    for (int s = 0; s <= t; ++s) {
      const float nk = pair[0][upto(t, s)], nb = pair[1][upto(t, s)];
      rt = fmaf(-nb, W[s], rt);
      zt = fmaf(nk, v[s], fmaf(-nb, X[s], zt));
    }
    record[VECTORS + (t * 4) * DK + i] = wt;
    record[VECTORS + (t * 4 + 1) * DK + i] = rt;
    float* slot = columns + (t * (COLS / 2) + in_group / 2) * 4 + (in_group & 1);
    slot[0] = v[t];
    slot[2] = xt;
    columns[CHUNK * COLS / 2 * 4 + t * COLS + in_group] = zt;
  }
  record[i] = run;
}

__device__ __forceinline__ void copy16(float* smem, const float* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Two packed fused multiply-adds, each rounded like a single one.
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
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

constexpr int SCAN_THREADS = 128, STAGES = 4;
constexpr int COPIED = COLUMNS + GROUP;           // floats of a record that one group of columns needs
constexpr int STAGE = (COPIED + 31) / 32 * 32;

// Sixteen lanes share a pair of columns of S, four rows each, in registers; a warp has two such pairs, a block eight.  A
// lane's partial sums of the chunk's W_t S and R_t S (two columns each) meet by halving: after the rounds over lane bits 3,
// 2, 1 and 0, lane p of the sixteen holds token p / 2, W where p is even and R where it is odd.  So that no value has to be
// chosen by lane, lane p walks the tokens and the two vectors in the order of (slot XOR its own number): the slot a lane
// keeps in a round is always the lower one.
__global__ void __launch_bounds__(SCAN_THREADS, 2)
delta_chunk_scan_kernel(const float* __restrict__ records, const Pass pass, const int* __restrict__ slots,
                        float* __restrict__ state, float* __restrict__ out, int heads, int dim, int max_slots) {
  tl::pdl_launch_dependents();
  extern __shared__ __align__(128) float smem[];  // [STAGES][STAGE]
  const int req = blockIdx.x, h = blockIdx.y, group = blockIdx.z, tid = threadIdx.x, lane = tid & 31;
  const int part = lane & 15, pair = (tid >> 5) * 2 + (lane >> 4);  // this lane's rows 4 part .., columns 2 pair and 2 pair + 1
  const int chunks = pass.chunks_of(req);
  int before = 0;
  for (int base = 0; base < req; base += 32) before += base + lane < req ? pass.chunks_of(base + lane) : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  // the request's tokens in this pass
  const int first = pass.req_indptr[req] + pass.lo * CHUNK, last = min(pass.req_indptr[req + 1], first + chunks * CHUNK);
  tl::pdl_wait();
  if (chunks == 0) return;
  const int hd = heads * dim, col = group * COLS + 2 * pair;
  const bool on = col < dim;  // (dim is even)
  const int slot = slots[req];
  const bool live = TL_DEBUG_OK(slot >= -1 && slot < max_slots, TL_DEBUG_SLOT, slot) && slot >= 0;
  if (!live) {  // padding: no state is touched
    if (part == 0 && on)
      for (int t = first; t < last; ++t) *reinterpret_cast<float2*>(out + (size_t)t * hd + h * dim + col) = make_float2(0.f, 0.f);
    return;
  }
  const float* source = records + ((size_t)before * heads + h) * RECORD;
  const size_t step = (size_t)heads * RECORD;
  auto fetch = [&](int c) {
    const float* from = source + (size_t)c * step;
    float* to = smem + (c % STAGES) * STAGE;
#pragma unroll
    for (int e = tid * 4; e < COPIED; e += SCAN_THREADS * 4) copy16(to + e, from + e + (e < COLUMNS ? 0 : group * GROUP));
    copies_commit();
  };
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c) {  // always STAGES - 1 groups in flight (some of them empty)
    if (c < chunks) fetch(c);
    else copies_commit();
  }
  // S in pairs of rows: S[column][rows 0 and 1, rows 2 and 3 of this lane's four]
  float* mine = state + ((size_t)slot * heads + h) * dim * dim;
  unsigned long long S[2][2];
  {
    float2 x[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = 4 * part + n;
      x[n] = on && i < dim ? *reinterpret_cast<const float2*>(mine + (size_t)i * dim + col) : make_float2(0.f, 0.f);
    }
    S[0][0] = pack2(x[0].x, x[1].x), S[0][1] = pack2(x[2].x, x[3].x);
    S[1][0] = pack2(x[0].y, x[1].y), S[1][1] = pack2(x[2].y, x[3].y);
  }
  const int my_token = part >> 1;
  const bool holds_out = part & 1;
  const int lane_at = VECTORS + my_token * 4 * DK + (part & 1) * DK;  // (token 0 XOR mine, vector 0 XOR mine)
  float* dst = out + (size_t)(first + my_token) * hd + h * dim + col;

  for (int c = 0; c < chunks; ++c) {
    copies_wait<STAGES - 2>();
    __syncthreads();  // this chunk has landed for every thread, and nobody reads the one before it any more
    if (c + STAGES - 1 < chunks) fetch(c + STAGES - 1);
    else copies_commit();
    float* stage = smem + (c % STAGES) * STAGE;
    // all of a chunk's vectors are requested before the first is used: with one warp on a scheduler the reads' latencies, one
    // after the other, would be what a chunk takes
    ulonglong2 seen[CHUNK][2], k[CHUNK], b[CHUNK];
#pragma unroll
    for (int j = 0; j < CHUNK; ++j)
#pragma unroll
      for (int x = 0; x < 2; ++x)
        seen[j][x] = *reinterpret_cast<const ulonglong2*>(stage + VECTORS + ((lane_at - VECTORS) ^ (j * 4 * DK | x * DK)) + 4 * part);
#pragma unroll
    for (int t = 0; t < CHUNK; ++t) {
      k[t] = *reinterpret_cast<const ulonglong2*>(stage + VECTORS + (t * 4 + 2) * DK + 4 * part);
      b[t] = *reinterpret_cast<const ulonglong2*>(stage + VECTORS + (t * 4 + 3) * DK + 4 * part);
    }
    const ulonglong2 decay = *reinterpret_cast<const ulonglong2*>(stage + 4 * part);
    float sum[CHUNK][2][2];  // [token slot][vector slot][column]
#pragma unroll
    for (int j = 0; j < CHUNK; ++j)
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 s = unpack2(fma2(seen[j][x].y, S[e][1], mul2(seen[j][x].x, S[e][0])));
          sum[j][x][e] = s.x + s.y;
        }
#pragma unroll
    for (int n = CHUNK / 2; n > 0; n >>= 1)
#pragma unroll
      for (int j = 0; j < n; ++j)
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int e = 0; e < 2; ++e) sum[j][x][e] += __shfl_xor_sync(0xffffffffu, sum[j + n][x][e], 2 * n);
    float2 mine_sum;
    mine_sum.x = sum[0][0][0] + __shfl_xor_sync(0xffffffffu, sum[0][1][0], 1);
    mine_sum.y = sum[0][0][1] + __shfl_xor_sync(0xffffffffu, sum[0][1][1], 1);
    float* columns = stage + COLUMNS;
    if (holds_out) {
      const float2 z = *reinterpret_cast<const float2*>(columns + CHUNK * COLS / 2 * 4 + my_token * COLS + 2 * pair);
      if (on && c * CHUNK + my_token < last - first) *reinterpret_cast<float2*>(dst) = make_float2(mine_sum.x + z.x, mine_sum.y + z.y);
    } else {  // y in place of X, for the sixteen lanes of these columns
      float2* x = reinterpret_cast<float2*>(columns + (my_token * (COLS / 2) + pair) * 4 + 2);
      *x = make_float2(mine_sum.x + x->x, mine_sum.y + x->y);
    }
    dst += (size_t)CHUNK * hd;
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 2; ++e) S[e][0] = mul2(decay.x, S[e][0]), S[e][1] = mul2(decay.y, S[e][1]);
    float4 vy[CHUNK];
#pragma unroll
    for (int t = 0; t < CHUNK; ++t) vy[t] = *reinterpret_cast<const float4*>(columns + (t * (COLS / 2) + pair) * 4);
#pragma unroll
    for (int t = 0; t < CHUNK; ++t) {
      const unsigned long long v[2] = {pack2(vy[t].x, vy[t].x), pack2(vy[t].y, vy[t].y)};
      const unsigned long long y[2] = {pack2(-vy[t].z, -vy[t].z), pack2(-vy[t].w, -vy[t].w)};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        S[e][0] = fma2(k[t].x, v[e], fma2(b[t].x, y[e], S[e][0]));
        S[e][1] = fma2(k[t].y, v[e], fma2(b[t].y, y[e], S[e][1]));
      }
    }
  }
  if (on) {
    const float2 a0 = unpack2(S[0][0]), a1 = unpack2(S[0][1]), b0 = unpack2(S[1][0]), b1 = unpack2(S[1][1]);
    const float2 x[4] = {make_float2(a0.x, b0.x), make_float2(a0.y, b0.y), make_float2(a1.x, b1.x), make_float2(a1.y, b1.y)};
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = 4 * part + n;
      if (i < dim) *reinterpret_cast<float2*>(mine + (size_t)i * dim + col) = x[n];
    }
  }
}

int sm_count() {
  static const int sms = [] {
    int device = 0, n = 0;
    return cudaGetDevice(&device) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && n > 0 ? n : 148;
  }();
  return sms;
}

}  // namespace

TL_DEBUG_READER(tl_delta_chunked_debug_error)

extern "C" {

// Tokens a chunk has, and the floats of a (chunk, head) that prepare leaves for the scan.
int tl_delta_chunk_tokens() { return CHUNK; }
int tl_delta_chunk_record() { return RECORD; }

// Chunks [lo, hi) of the requests of at least ``least`` tokens, ``chunks`` in all; the other requests' rows of ``out`` and their
// states are left as they are.  A step's chunks may go in several such passes, lo ascending: each continues from the states the
// one before it left, the bits are the same, and the scratch memory need not hold the whole step.
// proj rows, w2t, w0, a_bias as tl_delta_prepare's; state and out as tl_delta_scan's; records: chunks *
// heads * tl_delta_chunk_record() floats.  Head sizes up to 64, multiples of 4; everything starts on 16-byte boundaries.
int tl_delta_chunked(const float* proj, int proj_stride, const float* w2t, const float* w0, const float* a_bias,
                     const int* req_indptr, const int* slots, float* state, float* out, float* records, int requests, int chunks,
                     int lo, int hi, int least, int heads, int dim, int rank, int max_slots, cudaStream_t stream) {
  if (requests <= 0 || chunks <= 0) return 0;
  if (dim <= 0 || dim > DK || dim % 4 || heads <= 0 || heads > 65535 || rank <= 0 || rank > 1024 || least < 1 || lo < 0 || hi <= lo ||
      (((uintptr_t)state | (uintptr_t)out | (uintptr_t)records) & 15))
    return TL_ERR_UNSUPPORTED;
  const Pass pass{req_indptr, requests, least, lo, hi};
  tl::launch_kernel(delta_chunk_prepare_kernel, dim3(chunks, heads), DK, (size_t)CHUNK * rank * sizeof(float), stream, proj,
                    proj_stride, w2t, w0, a_bias, pass, records, heads, dim, rank);
  // (the blocks of requests without chunks leave at once; the others walk long enough that their places matter)
  tl::launch_apart<delta_chunk_scan_kernel>(dim3(requests, heads, (dim + COLS - 1) / COLS), SCAN_THREADS, true, sm_count(), 0,
                                            (size_t)STAGES * STAGE * sizeof(float), stream, (const float*)records, pass, slots, state,
                                            out, heads, dim, max_slots);
  return TL_LAUNCH_CHECK();
}

}  // extern "C"
