// Gated linear attention over long portions, chunk by chunk: the numbers of gla.cu's scan
//
//   S_t = diag(a_t) S_(t-1) + k_t v_t^T,      o_t = S_t^T q_t * qscale
//
// without its chain of tokens.  With the chunk's state S at its start and P(s, t) = prod of a_(s+1) .. a_t per channel,
//
//   o_t = (q_t * P(0, t))^T S + sum_(s <= t) A[t][s] v_s,     A[t][s] = sum_i q_t[i] k_s[i] P(s, t)[i],
//   S'  = diag(P(0, L)) S + sum_s (k_s * P(s, L)) v_s^T,
//
// so all chunks work at once except for one multiplication and addition of the state a chunk.  Everything is float32, and
// every decay between two tokens is a product of the decays between them (at most one each), never a quotient.
//
// Three kernels, blocks of 256 threads; a chunk is CHUNK tokens of one request:
//   state  a block a (chunk, head, VT value channels): the sum in S', and P(0, L);
//   carry  a thread four entries of a (request, head)'s state: walks the chunks, leaves each chunk's starting state in
//          place of its sum and the final state in the slot;
//   out    a block a (chunk, head, VT value channels): A, then both products of o.
// A is built in blocks of SUB x SUB tokens: on the diagonal token by token, each column's k times the running product of
// decays; below it as a product of q_t P(start of t's block, t) and k_s P(s, start of t's block).
//
// One request of 2,048 tokens, 16 heads of 64 x 128: 76 us for the three against 275 for the scan; 8 heads:
// 46 against 274.  Error against 64 bits, in 1e-7: 1.25 against the scan's 1.20 with decays sigmoid(x)^(1/12), 0.90 against 0.81 with
// ^(1/2), 2.35 against 3.9 with ^(1/200).  The order of a token's additions depends on where its chunk starts, so this form serves
// the bfloat16 engine; the float32 engine, whose logits do not depend on how a sequence is cut, keeps the scan.
#include "common.cuh"

namespace {

using namespace tl;

constexpr int CHUNK = 64, SUB = 16, DK = 64, LD = DK + 4;  // (rows of LD floats: eight rows' pieces fall into different banks)
constexpr int NT = 256;

__device__ __forceinline__ void copy16(void* smem, const void* gmem, bool on) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int bytes = on ? 16 : 0;  // 0: the 16 bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Two packed fused multiply-adds, each rounded like a single one.
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

struct Args {
  const float* proj;  // rows [q (H D) | k (H D) | v (H V) | ...]
  const float* decay;  // [tokens, H D]
  const int* req_indptr;
  const int* slots;
  float* state;   // [slots, H, D, V]
  float* out;     // [tokens, H V]
  float* sums;    // [chunks, H, D, V]: a chunk's sum, then its starting state
  float* decays;  // [chunks, H, DK]: P(0, L)
  int proj_stride, requests, heads, dim, vdim, max_slots, least;
  float qscale;
};

// Requests of ``least`` tokens and more are cut into chunks, in the order of the requests; the others have none here.
__device__ __forceinline__ int chunks_of(const Args& p, int req) {
  const int n = req < p.requests ? p.req_indptr[req + 1] - p.req_indptr[req] : 0;
  return n >= p.least ? (n + CHUNK - 1) / CHUNK : 0;
}
// The request and the first token and the number of tokens of chunk ``id``; every warp finds them by itself.
__device__ __forceinline__ bool find_chunk(const Args& p, int id, int& req, int& first, int& count) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < p.requests; base += 32) {
    const int mine = chunks_of(p, base + lane);
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int below = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += below;
    }
    const unsigned beyond = __ballot_sync(0xffffffffu, upto > id);
    if (beyond) {
      const int at = __ffs(beyond) - 1;
      const int before = __shfl_sync(0xffffffffu, upto - mine, at);
      req = base + at;
      first = p.req_indptr[req] + (id - before) * CHUNK;
      count = min(CHUNK, p.req_indptr[req + 1] - first);
      return true;
    }
    id -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

// Rows of a chunk into shared memory (zeros past its tokens and past ``dim``): [CHUNK][LD] from rows ``stride`` apart.
__device__ __forceinline__ void load_rows(float* dst, const float* src, long long stride, int count, int dim) {
  for (int e = threadIdx.x; e < CHUNK * DK / 4; e += NT) {
    const int t = e / (DK / 4), c = (e % (DK / 4)) * 4;
    const bool on = t < count && c < dim;
    copy16(dst + t * LD + c, on ? src + t * stride + c : src, on);
  }
}
template <int VT>
__device__ __forceinline__ void load_tile(float* dst, const float* src, long long stride, int rows, int cols) {
  for (int e = threadIdx.x; e < CHUNK * VT / 4; e += NT) {
    const int t = e / (VT / 4), c = (e % (VT / 4)) * 4;
    const bool on = t < rows && c < cols;
    copy16(dst + t * VT + c, on ? src + t * stride + c : src, on);
  }
}
// Decays past the chunk's tokens and past ``dim`` count as one.
__device__ __forceinline__ void ones_past(float* a, int count, int dim) {
  if (count == CHUNK && dim == DK) return;
  for (int e = threadIdx.x; e < CHUNK * DK; e += NT) {
    const int t = e / DK, c = e % DK;
    if (t >= count || c >= dim) a[t * LD + c] = 1.f;
  }
}

// sum[4 rows][8 columns] += x[rows][n] y[n][columns], n a multiple of 16, each sixteen products on their own first (one chain
// of 128 additions rounds further off than the scan's short ones).  x: four rows from ``x`` on, LD apart; y: rows of VT floats,
// the thread's columns are 4 jg and VT / 2 + 4 jg.  CAUSAL: of the last sixteen products row r takes those up to number
// ``last`` + r only (``last`` a multiple of 4): a factor behind them is never multiplied, not even with zero, which would make
// NaN of an infinite one.
template <int VT, bool CAUSAL>
__device__ __forceinline__ void tile_fma(float2 (&sum)[4][4], const float* x, const float* y, int n, int jg, int last = 12) {
#pragma unroll 1
  for (int k = 0; k < n; k += 16) {
    unsigned long long acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0ull;
    const int stop = CAUSAL && k + 16 >= n ? last : 16;
#pragma unroll
    for (int kk = 0; kk < 16; kk += 4) {
      if (CAUSAL && kk > stop) break;
      float4 a[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4*>(x + r * LD + k + kk);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(y + (k + kk + e) * VT + 4 * jg);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(y + (k + kk + e) * VT + VT / 2 + 4 * jg);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (CAUSAL && e > r && kk == stop) continue;
          const unsigned long long s = twice(e == 0 ? a[r].x : e == 1 ? a[r].y : e == 2 ? a[r].z : a[r].w);
          fma2(acc[r][0], s, b0.x);
          fma2(acc[r][1], s, b0.y);
          fma2(acc[r][2], s, b1.x);
          fma2(acc[r][3], s, b1.y);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 v = unpack2(acc[r][j]);
        sum[r][j].x += v.x;
        sum[r][j].y += v.y;
      }
  }
}

template <int VT>
__global__ void __launch_bounds__(NT, 2)
gla_chunk_state_kernel(const Args p) {
  tl::pdl_launch_dependents();
  extern __shared__ __align__(16) float smem[];
  float* k = smem;              // [DK][LD] after the transposition: channel by token
  float* a = k + CHUNK * LD;
  float* v = a + CHUNK * LD;    // [CHUNK][VT]
  __shared__ float segment[CHUNK / SUB][DK];
  const int h = blockIdx.y, col0 = blockIdx.z * VT, tid = threadIdx.x;
  int req, first, count;
  const bool found = find_chunk(p, blockIdx.x, req, first, count);
  tl::pdl_wait();
  if (!found || p.slots[req] < 0) return;
  const float* row = p.proj + (size_t)first * p.proj_stride;
  load_rows(k, row + (size_t)p.heads * p.dim + h * p.dim, p.proj_stride, count, p.dim);
  load_rows(a, p.decay + ((size_t)first * p.heads + h) * p.dim, (long long)p.heads * p.dim, count, p.dim);
  copies_commit();
  load_tile<VT>(v, row + (size_t)2 * p.heads * p.dim + h * p.vdim + col0, p.proj_stride, count, p.vdim - col0);
  copies_commit();
  copies_wait<1>();
  __syncthreads();
  ones_past(a, count, p.dim);
  __syncthreads();
  // k_s P(s, L), kept in registers and written back channel by token
  const int c = tid % DK, seg = tid / DK;
  float mine[SUB], run = 1.f;
#pragma unroll
  for (int j = SUB - 1; j >= 0; --j) {
    mine[j] = k[(seg * SUB + j) * LD + c] * run;
    run *= a[(seg * SUB + j) * LD + c];
  }
  segment[seg][c] = run;
  __syncthreads();
  float after = 1.f;
  for (int s = CHUNK / SUB - 1; s > seg; --s) after *= segment[s][c];
#pragma unroll
  for (int j = 0; j < SUB; j += 4)
    *reinterpret_cast<float4*>(k + c * LD + seg * SUB + j) =
        make_float4(mine[j] * after, mine[j + 1] * after, mine[j + 2] * after, mine[j + 3] * after);
  if (seg == 0 && blockIdx.z == 0) p.decays[((size_t)blockIdx.x * p.heads + h) * DK + c] = run * after;
  copies_wait<0>();
  __syncthreads();
  constexpr int JG = VT / 8;
  const int jg = tid % JG, ig = tid / JG;
  if (ig >= DK / 4) return;
  float2 acc[4][4] = {};
  tile_fma<VT, false>(acc, k + ig * 4 * LD, v, (count + 15) / 16 * 16, jg);
  float* dst = p.sums + ((size_t)blockIdx.x * p.heads + h) * p.dim * p.vdim + col0;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ig * 4 + r;
    if (i >= p.dim) break;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int j = half * (VT / 2) + 4 * jg;
      if (col0 + j < p.vdim) {
        const float2 lo = acc[r][2 * half], hi = acc[r][2 * half + 1];
        *reinterpret_cast<float4*>(dst + (size_t)i * p.vdim + j) = make_float4(lo.x, lo.y, hi.x, hi.y);
      }
    }
  }
}

__global__ void __launch_bounds__(NT)
gla_chunk_carry_kernel(const Args p) {
  tl::pdl_launch_dependents();
  const int req = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31;
  int before = 0;
  for (int base = 0; base < req; base += 32) before += base + lane < req ? chunks_of(p, base + lane) : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  const int chunks = chunks_of(p, req);
  const int e = (blockIdx.z * NT + threadIdx.x) * 4, size = p.dim * p.vdim;
  tl::pdl_wait();
  const int slot = p.slots[req];
  const bool live = TL_DEBUG_OK(slot >= -1 && slot < p.max_slots, TL_DEBUG_SLOT, slot) && slot >= 0;
  if (!live || chunks == 0 || e >= size) return;
  const int i = e / p.vdim;
  float* mine = p.state + ((size_t)slot * p.heads + h) * size + e;
  float* sum = p.sums + ((size_t)before * p.heads + h) * size + e;
  const float* decay = p.decays + ((size_t)before * p.heads + h) * DK + i;
  const size_t step = (size_t)p.heads * size, decay_step = (size_t)p.heads * DK;
  float4 S = *reinterpret_cast<const float4*>(mine);
  constexpr int AHEAD = 8;  // chunks requested at once
  for (int c = 0; c < chunks; c += AHEAD) {
    float4 f[AHEAD];
    float d[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (c + j < chunks) {
        f[j] = *reinterpret_cast<const float4*>(sum + (c + j) * step);
        d[j] = decay[(c + j) * decay_step];
      }
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (c + j < chunks) {
        *reinterpret_cast<float4*>(sum + (c + j) * step) = S;
        S = make_float4(fmaf(d[j], S.x, f[j].x), fmaf(d[j], S.y, f[j].y), fmaf(d[j], S.z, f[j].z), fmaf(d[j], S.w, f[j].w));
      }
  }
  *reinterpret_cast<float4*>(mine) = S;
}

template <int VT>
__global__ void __launch_bounds__(NT, 2)
gla_chunk_out_kernel(const Args p) {
  tl::pdl_launch_dependents();
  extern __shared__ __align__(16) float smem[];
  float* A = smem;              // [CHUNK][LD] scores
  float* q = A + CHUNK * LD;
  float* k = q + CHUNK * LD;
  float* a = k + CHUNK * LD;
  float* v = a + CHUNK * LD;    // [CHUNK][VT]
  float* S = k;                 // [DK][VT], in place of k and a once the scores are there
  static_assert(2 * CHUNK * LD >= DK * VT, "the starting state fits where k and a were");
  __shared__ float segment[CHUNK / SUB][DK];
  const int h = blockIdx.y, col0 = blockIdx.z * VT, tid = threadIdx.x;
  const int hv = p.heads * p.vdim;
  int req, first, count;
  const bool found = find_chunk(p, blockIdx.x, req, first, count);
  tl::pdl_wait();
  if (!found) return;
  float* out = p.out + (size_t)first * hv + h * p.vdim + col0;
  if (p.slots[req] < 0) {  // padding: no state is read
    for (int e = tid; e < count * VT; e += NT)
      if (col0 + e % VT < p.vdim) out[(size_t)(e / VT) * hv + e % VT] = 0.f;
    return;
  }
  const float* row = p.proj + (size_t)first * p.proj_stride;
  load_rows(q, row + h * p.dim, p.proj_stride, count, p.dim);
  load_rows(k, row + (size_t)p.heads * p.dim + h * p.dim, p.proj_stride, count, p.dim);
  load_rows(a, p.decay + ((size_t)first * p.heads + h) * p.dim, (long long)p.heads * p.dim, count, p.dim);
  copies_commit();
  load_tile<VT>(v, row + (size_t)2 * p.heads * p.dim + h * p.vdim + col0, p.proj_stride, count, p.vdim - col0);
  copies_commit();
  copies_wait<1>();
  __syncthreads();
  ones_past(a, count, p.dim);
  __syncthreads();

  // ---- scores of tokens of one SUB: four lanes a column s, 16 channels each, t ascending
  {
    const int part = tid & 3, s = tid >> 2;
    float w[DK / 4];
#pragma unroll
    for (int n = 0; n < DK / 16; ++n) {
      const float4 x = *reinterpret_cast<const float4*>(k + s * LD + 16 * n + 4 * part);
      w[4 * n] = x.x; w[4 * n + 1] = x.y; w[4 * n + 2] = x.z; w[4 * n + 3] = x.w;
    }
    for (int step = 0; step < SUB; ++step) {  // the same number of steps for every lane: the shuffles are the warp's
      const int t = s / SUB * SUB + step;
      float sum = 0.f;
      if (t > s) {
#pragma unroll
        for (int n = 0; n < DK / 16; ++n) {
          const float4 x = *reinterpret_cast<const float4*>(a + t * LD + 16 * n + 4 * part);
          w[4 * n] *= x.x; w[4 * n + 1] *= x.y; w[4 * n + 2] *= x.z; w[4 * n + 3] *= x.w;
        }
      }
      if (t >= s) {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int n = 0; n < DK / 16; ++n) {
          const float4 x = *reinterpret_cast<const float4*>(q + t * LD + 16 * n + 4 * part);
          s0 = fmaf(x.x, w[4 * n], s0);
          s1 = fmaf(x.y, w[4 * n + 1], s1);
          s0 = fmaf(x.z, w[4 * n + 2], s0);
          s1 = fmaf(x.w, w[4 * n + 3], s1);
        }
        sum = s0 + s1;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if (part == 0) A[t * LD + s] = sum;  // (zero above the diagonal)
    }
  }
  __syncthreads();

  // ---- q_t P(start of its SUB, t) and k_s P(s, end of its SUB), in place
  const int c = tid % DK, seg = tid / DK;
  {
    float run = 1.f;
#pragma unroll
    for (int j = 0; j < SUB; ++j) {
      run *= a[(seg * SUB + j) * LD + c];
      q[(seg * SUB + j) * LD + c] *= run;
    }
    segment[seg][c] = run;
    run = 1.f;
#pragma unroll
    for (int j = SUB - 1; j >= 0; --j) {
      k[(seg * SUB + j) * LD + c] *= run;
      run *= a[(seg * SUB + j) * LD + c];
    }
  }
  __syncthreads();

  // ---- scores below the diagonal blocks: rows of SUB number b against all earlier tokens, whose k meanwhile carry the
  // decays up to the start of b
#pragma unroll 1
  for (int b = 1; b < CHUNK / SUB; ++b) {
    if (b > 1) {
      if (seg < b - 1) {
        const float more = segment[b - 1][c];
#pragma unroll
        for (int j = 0; j < SUB; ++j) k[(seg * SUB + j) * LD + c] *= more;
      }
      __syncthreads();
    }
    // 16 x 16 b scores, two neighbouring rows of a column a thread and turn
    for (int o = tid; o < SUB / 2 * b * SUB; o += NT) {
      const int s = o % (b * SUB), t = b * SUB + o / (b * SUB) * 2;
      float s0 = 0.f, s1 = 0.f, r0 = 0.f, r1 = 0.f;
#pragma unroll
      for (int n = 0; n < DK; n += 4) {
        const float4 x = *reinterpret_cast<const float4*>(k + s * LD + n);
        const float4 y = *reinterpret_cast<const float4*>(q + t * LD + n), z = *reinterpret_cast<const float4*>(q + (t + 1) * LD + n);
        s0 = fmaf(x.x, y.x, s0); s1 = fmaf(x.y, y.y, s1); s0 = fmaf(x.z, y.z, s0); s1 = fmaf(x.w, y.w, s1);
        r0 = fmaf(x.x, z.x, r0); r1 = fmaf(x.y, z.y, r1); r0 = fmaf(x.z, z.z, r0); r1 = fmaf(x.w, z.w, r1);
      }
      A[t * LD + s] = s0 + s1;
      A[(t + 1) * LD + s] = r0 + r1;
    }
    __syncthreads();
  }
  // the starting state takes the place of k and a
  load_tile<VT>(S, p.sums + ((size_t)blockIdx.x * p.heads + h) * p.dim * p.vdim + col0, p.vdim, p.dim, p.vdim - col0);
  copies_commit();
  {
    float earlier = 1.f;
    for (int s = 0; s < seg; ++s) earlier *= segment[s][c];
#pragma unroll
    for (int j = 0; j < SUB; ++j) q[(seg * SUB + j) * LD + c] *= earlier;
  }
  copies_wait<0>();
  __syncthreads();

  constexpr int JG = VT / 8;
  const int jg = tid % JG, tg = tid / JG;
  if (tg >= CHUNK / 4 || tg * 4 >= count) return;
  float2 acc[4][4] = {};
  tile_fma<VT, false>(acc, q + tg * 4 * LD, S, DK, jg);
  tile_fma<VT, true>(acc, A + tg * 4 * LD, v, (tg * 4 / SUB + 1) * SUB, jg, tg * 4 % SUB);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int t = tg * 4 + r;
    if (t >= count) break;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int j = half * (VT / 2) + 4 * jg;
      if (col0 + j < p.vdim) {
        const float2 lo = acc[r][2 * half], hi = acc[r][2 * half + 1];
        *reinterpret_cast<float4*>(out + (size_t)t * hv + j) =
            make_float4(lo.x * p.qscale, lo.y * p.qscale, hi.x * p.qscale, hi.y * p.qscale);
      }
    }
  }
}

template <int VT>
int launch(const Args& p, int chunks, cudaStream_t stream) {
  constexpr int STATE = (2 * CHUNK * LD + CHUNK * VT) * 4, OUT = (4 * CHUNK * LD + CHUNK * VT) * 4;
  static_assert(2 * (OUT + 2048) <= 228 * 1024, "two blocks an SM");
  static const cudaError_t configured = [] {
    const cudaError_t e = cudaFuncSetAttribute(gla_chunk_state_kernel<VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, STATE);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(gla_chunk_out_kernel<VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT);
  }();
  if (configured != cudaSuccess) return (int)configured;
  const dim3 grid(chunks, p.heads, (p.vdim + VT - 1) / VT);
  tl::launch_kernel(gla_chunk_state_kernel<VT>, grid, NT, STATE, stream, p);
  tl::launch_kernel(gla_chunk_carry_kernel, dim3(p.requests, p.heads, (p.dim * p.vdim / 4 + NT - 1) / NT), NT, 0, stream, p);
  tl::launch_kernel(gla_chunk_out_kernel<VT>, grid, NT, OUT, stream, p);
  return TL_LAUNCH_CHECK();
}

}  // namespace

TL_DEBUG_READER(tl_gla_chunked_debug_error)

extern "C" {

// Tokens a chunk has.
int tl_gla_chunk_tokens() { return CHUNK; }

// The requests of at least ``least`` tokens, which have ``chunks`` chunks in all; the other requests' rows of ``out`` and
// their states are left as they are.  workspace: chunks * heads * (dim * vdim + 64) floats.  Head sizes up to 64 (keys) and
// 256 (values), multiples of 4; all rows start on 16-byte boundaries.
int tl_gla_chunked(const float* proj, int proj_stride, const float* decay, const int* req_indptr, const int* slots, float* state,
                   float* out, float* workspace, int requests, int chunks, int least, int heads, int dim, int vdim, int max_slots,
                   float qscale, cudaStream_t stream) {
  if (requests <= 0 || chunks <= 0) return 0;
  const uintptr_t all = (uintptr_t)proj | (uintptr_t)decay | (uintptr_t)state | (uintptr_t)out | (uintptr_t)workspace;
  if (dim <= 0 || dim > DK || dim % 4 || vdim <= 0 || vdim > 256 || vdim % 4 || proj_stride % 4 || (all & 15) || heads <= 0 ||
      heads > 65535 || least < 1)
    return TL_ERR_UNSUPPORTED;
  const Args p{proj, decay, req_indptr, slots, state, out, workspace, workspace + (size_t)chunks * heads * dim * vdim,
               proj_stride, requests, heads, dim, vdim, max_slots, least, qscale};
  return vdim <= 64 ? launch<64>(p, chunks, stream) : launch<128>(p, chunks, stream);
}

}  // extern "C"
