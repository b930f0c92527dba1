// Paged causal grouped-query attention for any batch of (request, next tokens):
// prompt portions with cached context before them and single decoded tokens alike.
// One warp per (token, query head); keys are visited in tiles of 32 consecutive
// ABSOLUTE positions (tile edges at multiples of 32), so the order of every sum
// depends only on the token's position and window, never on how the sequence was cut
// into steps, on the batch, or on the pages used.  Scores, softmax and the weighted
// sum are float32; T is the storage type of queries, pages and output.
//
// Options: ``softcap`` > 0 bounds a score, s <- softcap tanh(s / softcap); ``sink`` adds one to the
// softmax's denominator (a key of score 0 that has no value), or with ``sink_values`` exp(sink_values[head]); ``gate`` (float32 rows) multiplies the
// output element by element with sigmoid(gate).
//
// ``keep`` > 0: the first ``keep`` positions of the sequence are visible beside the window (their tiles come first).
// ``chunks`` = nkv: a query row spans the keys of ALL KV heads, [nh][nkv][d], and a head's score is the sum over them
// (scores mixed across the heads, folded into the queries; see csrc/qkv_prepare.cu); 1: the head's own KV head alone.
// ``v_cols``: how many entries of a value row are written for a head (the cache rows may be padded).
//
// Two more kernels take the 32-bit rows of head_dim up to 128 (a multiple of 4) whose keys lie in one window and whose heads
// read one KV head each (``in_chunks`` below; a rule on the layer alone, so a request never changes between the orders):
//   attention_f32_single_kernel   requests that bring one token, or few: a block a (token, head), eight warps, each a chunk of keys;
//   attention_f32_rows_kernel     tokens that stand beside many others of their request: 32 packed (token, head) rows of a KV
//                                 head share the key and value tiles in shared memory.
// Both cut the keys into CHUNKS of 64 absolute positions: a chunk is an online softmax of its own over its tiles of 32 keys,
// and the chunks are merged in ascending order.  So the order of every sum still depends on the position and window
// only, and a long context no longer is one chain: measurements at the kernels.
//
// attention_generic_kernel is the 32-bit kernel of all other forms and the any-size bfloat16 kernel (head_dim up to 256: keys are
// read eight entries at a time where head_dim and the query stride are multiples of 8, one at a
// time otherwise; any head counts, any page size).
//
// Reference counterparts: forward_ragged_attention_kernel and
// forward_slot_attention_decode_kernel, v10_triton_paged_gqa/kernel/gqa.py:5-228
// (query head h reads KV head h // g, scale head_dim^-0.5, key allowed iff
// key_pos <= query_pos, online softmax, acc / l).
#include <limits.h>
#include <math.h>

#include "common.cuh"

namespace {

using namespace tl;

constexpr int WARPS = 4;
constexpr int MAX_D = 256;

template <typename T>
__global__ void __launch_bounds__(WARPS * 32)
attention_generic_kernel(const T* __restrict__ q, int q_stride, const T* __restrict__ pages,
                         const int* __restrict__ block_table, int table_width,
                         const int* __restrict__ token_req, const int* __restrict__ positions,
                         T* __restrict__ out, int out_stride, int tokens, int nh, int nkv, int d,
                         int page_size, int window, float scale, int num_pages, float softcap, int sink,
                         const float* __restrict__ sink_values, const float* __restrict__ gate, int gate_stride, int wide,
                         int keep, int chunks, int v_cols) {
  tl::pdl_wait();               // everything before us in the stream is complete and visible
  tl::pdl_launch_dependents();  // the next kernel may start its own prologue

  extern __shared__ __align__(16) float all_queries[];  // [WARPS][chunks d]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * WARPS + warp;
  if (item >= (long long)tokens * nh) return;
  const int t = (int)(item / nh), h = (int)(item % nh);
  const int kvh = h / (nh / nkv);
  const int pos = positions[t];
  const int lo = first_key(pos, window);
  const int* table = block_table + (size_t)token_req[t] * table_width;

  const int q_len = chunks * d;
  float* qs = all_queries + warp * q_len;
  const T* qrow = q + (size_t)t * q_stride + (size_t)h * q_len;
  for (int i = lane; i < q_len; i += 32) qs[i] = to_float(qrow[i]);
  __syncwarp();

  const size_t page_elems = (size_t)2 * nkv * page_size * d;
  const size_t k_off = chunks > 1 ? 0 : (size_t)kvh * page_size * d;
  const size_t head_step = (size_t)page_size * d;  // from a key to the next KV head's
  const size_t v_off = ((size_t)nkv + kvh) * page_size * d;

  // the sink is a key of a given score (0, or the head's own number) and no value that every query sees: the running
  // maximum starts at that score with a weight of exp(0) in the denominator
  float m = sink ? (sink_values ? sink_values[h] : 0.f) : -INFINITY, l = sink ? 1.f : 0.f;
  float acc[MAX_D / 32];
#pragma unroll
  for (int c = 0; c < MAX_D / 32; ++c) acc[c] = 0.f;

  // tiles of kept first positions that lie wholly before the window's first tile, then the window's
  const int window_start = lo & ~31;
  const int kept_end = keep < window_start ? (keep + 31) & ~31 : window_start;
  for (int start = kept_end > 0 ? 0 : window_start; start <= pos;
       start = start + 32 == kept_end ? window_start : start + 32) {
    const int key = start + lane;
    const bool valid = (key >= lo || key < keep) && key <= pos;
    float s = -INFINITY;
    size_t row_off = 0;
    if (valid) {
      int page = 0;  // a key whose table entry fails a debug-build check is read from the reserved page 0
      if (TL_DEBUG_OK(key / page_size < table_width, TL_DEBUG_POSITION, key)) page = table[key / page_size];
      if (!TL_DEBUG_OK(page >= 0 && page < num_pages, TL_DEBUG_PAGE, page)) page = 0;
      row_off = (size_t)page * page_elems + (size_t)(key % page_size) * d;
      const T* krow = pages + row_off + k_off;
      float dot = 0.f;
      for (int c = 0; c < chunks; ++c, krow += head_step) {
        const float* qc = qs + c * d;
        if (wide) {
          for (int i = 0; i < d; i += 8) {
            float kv[8];
            load8(krow + i, kv);
#pragma unroll
            for (int j = 0; j < 8; ++j) dot = fmaf(qc[i + j], kv[j], dot);
          }
        } else {  // the same order of additions, one entry at a time
          for (int i = 0; i < d; ++i) dot = fmaf(qc[i], to_float(krow[i]), dot);
        }
      }
      s = dot * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    }
    const float new_m = fmaxf(m, warp_max(s));
    const float corr = expf(m - new_m);  // first tile: exp(-inf) = 0
    const float p = valid ? expf(s - new_m) : 0.f;
    l = l * corr + warp_sum(p);
    m = new_m;
#pragma unroll
    for (int c = 0; c < MAX_D / 32; ++c) acc[c] *= corr;
    const int first = start >= keep && lo > start ? lo - start : 0;  // (a lane without a key has weight 0 and is skipped)
    const int last = pos - start < 31 ? pos - start : 31;
    for (int j = first; j <= last; ++j) {
      if (keep && !__shfl_sync(0xffffffffu, (int)valid, j)) continue;
      const float pj = __shfl_sync(0xffffffffu, p, j);
      const size_t off = __shfl_sync(0xffffffffu, (unsigned long long)row_off, j);
      const T* vrow = pages + off + v_off;
#pragma unroll
      for (int c = 0; c < MAX_D / 32; ++c) {
        const int i = lane + 32 * c;
        if (i < d) acc[c] = fmaf(pj, to_float(vrow[i]), acc[c]);
      }
    }
  }
  T* orow = out + (size_t)t * out_stride + (size_t)h * v_cols;
  const float inv = 1.f / l;
#pragma unroll
  for (int c = 0; c < MAX_D / 32; ++c) {
    const int i = lane + 32 * c;
    if (i < v_cols) {
      float v = acc[c] * inv;
      if (gate) v *= 1.f / (1.f + expf(-gate[(size_t)t * gate_stride + (size_t)h * d + i]));
      orow[i] = from_float<T>(v);
    }
  }
}

// ------------------------------------------------------------------------------------- float32, keys in chunks of 64
constexpr int CHUNK_KEYS = 64;

// An online softmax over some keys: largest score, weights' sum, and this lane's entries of the weighted sum of values.
template <int VE> struct Softmax {
  float m, l, acc[VE];
  // Of a chunk whose scores are all -inf nothing remains; the others' keys count as ever.
  static __device__ __forceinline__ float finite(float top) { return top == -INFINITY ? 0.f : top; }
  __device__ __forceinline__ void clear() {
    m = -INFINITY;
    l = 0.f;
#pragma unroll
    for (int i = 0; i < VE; ++i) acc[i] = 0.f;
  }
  // A tile of 32 keys, one a lane, at least one of them valid, ``top`` their largest score: the lane's weight; then, with
  // the sum of the tile's weights, the state behind the tile.
  __device__ __forceinline__ float weight(float s, float top, bool valid) const { return valid ? expf(s - finite(fmaxf(m, top))) : 0.f; }
  __device__ __forceinline__ void rescale(float top, float sum) {
    const float new_m = fmaxf(m, top), corr = expf(m - finite(new_m));
    l = fmaf(l, corr, sum);
    m = new_m;
#pragma unroll
    for (int i = 0; i < VE; ++i) acc[i] = __fmul_rn(acc[i], corr);
  }
  // Takes the keys of a later chunk in.
  __device__ __forceinline__ void merge(float m2, float l2, const float (&acc2)[VE]) {
    const float new_m = fmaxf(m, m2), a = expf(m - finite(new_m)), b = expf(m2 - finite(new_m));
    l = fmaf(l, a, __fmul_rn(l2, b));
#pragma unroll
    for (int i = 0; i < VE; ++i) acc[i] = fmaf(acc[i], a, __fmul_rn(acc2[i], b));
    m = new_m;
  }
};

__device__ __forceinline__ float scored(float dot, float scale, float softcap) {
  const float s = __fmul_rn(dot, scale);
  return softcap > 0.f ? __fmul_rn(softcap, tanhf(s / softcap)) : s;
}

// What both kernels are given.
struct ChunkArgs {
  const float* q;
  const float* pages;
  const int* block_table;
  const int* token_req;
  const int* positions;
  float* out;
  const float* sink_values;
  const float* gate;
  int q_stride, table_width, out_stride, tokens, nh, nkv, d, page_size, window, num_pages, sink, gate_stride, v_cols, all_few;
  float scale, softcap;
};

__device__ __forceinline__ size_t key_row(const ChunkArgs& p, const int* table, int key, int kvh) {
  int page = 0;  // a key whose table entry fails a debug-build check is read from the reserved page 0
  if (TL_DEBUG_OK(key / p.page_size < p.table_width, TL_DEBUG_POSITION, key)) page = table[key / p.page_size];
  if (!TL_DEBUG_OK(page >= 0 && page < p.num_pages, TL_DEBUG_PAGE, page)) page = 0;
  return (((size_t)page * 2 * p.nkv + kvh) * p.page_size + key % p.page_size) * p.d;
}
// Requests that bring up to this many tokens go token by token: they fill too little of the packed rows of a block, which takes
// its requests one after the other.  32 requests of 2 tokens behind 1,000 at 8 heads of 64 with a KV head each: 59 us, packed 938
// (one warp a (token, head): 670).
__host__ __device__ __forceinline__ int few_tokens(int group) { return group < 8 ? 8 / group : 1; }
// Whether the request of token t brings at most ``few`` <= 8 tokens to the step (asked by all lanes of a warp).
__device__ __forceinline__ bool among_few(const ChunkArgs& p, int t, int few) {
  const int u = t + (int)(threadIdx.x & 31) - 15;  // the neighbours; lane 15 has t itself
  const bool there = u >= 0 && u < p.tokens;
  const int req = there ? p.token_req[u] : 0, mine = __shfl_sync(0xffffffffu, req, 15);
  const unsigned same = __ballot_sync(0xffffffffu, there && req == mine);
  return __ffs(~(same >> 15)) - 1 + __clz(~(same << 17)) <= few;  // the ones from bit 15 up and those right below it
}
__device__ __forceinline__ void write_out(const ChunkArgs& p, int t, int h, int i, float acc, float inv) {
  if (i >= p.v_cols) return;
  float v = acc * inv;
  if (p.gate) v *= 1.f / (1.f + expf(-p.gate[(size_t)t * p.gate_stride + (size_t)h * p.d + i]));
  p.out[(size_t)t * p.out_stride + (size_t)h * p.v_cols + i] = v;
}

// Bound by the latency of its walk: table entry, key and value rows, weights.  Eight warps take a chunk of 64 keys each, so
// 700 keys are two rounds and not 22 tiles in a row, and a tile's values are requested with its keys: a step of 8 requests of up
// to 700 keys at 14 heads of 64 takes 17 us a layer, 47 with the values requested behind the scores, eight keys at a
// time (one warp a (token, head): 440).  Up to 4 chunks leave warps of such a block idle: in a grid of
// more than two waves (PACK) it then takes 2, 4 or 8 heads and the blocks of the others leave at once.  64 requests of 40 keys at
// 28 heads of 128: 27 us, a head a block 46; one such request 14 and 7.4.
constexpr int SINGLE_WARPS = 8;

template <int DP, bool PACK>
__global__ void __launch_bounds__(SINGLE_WARPS * 32, 2) attention_f32_single_kernel(const ChunkArgs p) {
  tl::pdl_wait();
  tl::pdl_launch_dependents();
  constexpr int VE = DP / 32, BATCH = 64 / VE;  // keys whose values are requested together
  __shared__ __align__(16) float qs[PACK ? SINGLE_WARPS : 1][DP];  // of the block's heads
  __shared__ float parts[2][SINGLE_WARPS][DP + 2];      // a chunk's acc, m, l; two rounds
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x / p.nh, h0 = blockIdx.x % p.nh, d = p.d;
  if (!p.all_few && !among_few(p, t, few_tokens(p.nh / p.nkv))) return;
  // what does not hang on the position is requested before it
  const int pos = p.positions[t], req = p.token_req[t];
  const float* q_rows = p.q + (size_t)t * p.q_stride;
  const float first_q = threadIdx.x < d ? q_rows[(size_t)h0 * d + threadIdx.x] : 0.f;
  if (threadIdx.x < DP) qs[0][threadIdx.x] = first_q;
  const int lo = first_key(pos, p.window);
  const int chunks = pos / CHUNK_KEYS - lo / CHUNK_KEYS + 1;
  // warps a head, a power of two: with fewer than eight one round is all
  const int per_log2 = !PACK || chunks > 4 ? 3 : (chunks > 2 ? 2 : chunks - 1), per = 1 << per_log2, heads = SINGLE_WARPS >> per_log2;
  if (h0 & (heads - 1)) return;
  const int local = PACK ? warp >> per_log2 : 0, h = h0 + local;  // this warp's head of the block's
  const int kvh = h / (p.nh / p.nkv);
  const int* table = p.block_table + (size_t)req * p.table_width;
  for (int e = DP + threadIdx.x; e < heads * DP; e += SINGLE_WARPS * 32) {
    const int head = h0 + e / DP, i = e % DP;
    qs[e / DP][i] = i < d && head < p.nh ? q_rows[(size_t)head * d + i] : 0.f;
  }
  __syncthreads();
  const float* my_q = qs[local];
  const size_t values = (size_t)p.nkv * p.page_size * d;  // from a key to its value
  auto nothing_yet = [&](int head) {
    Softmax<1> s;
    s.clear();
    if (p.sink) {
      s.m = p.sink_values ? p.sink_values[head] : 0.f;
      s.l = 1.f;
    }
    return s;
  };
  const int i = threadIdx.x;  // the entry this thread merges where the block has one head
  Softmax<1> total = nothing_yet(h0);
  int buf = 0;
  for (int first = lo / CHUNK_KEYS; first <= pos / CHUNK_KEYS; first += per, buf ^= 1) {
    const int chunk = first + (PACK ? warp & (per - 1) : warp);
    if (chunk <= pos / CHUNK_KEYS && h < p.nh) {
      Softmax<VE> part;
      part.clear();
      for (int start = chunk * CHUNK_KEYS; start < (chunk + 1) * CHUNK_KEYS && start <= pos; start += 32) {
        if (start + 31 < lo) continue;
        const int key = start + lane;
        const bool valid = key >= lo && key <= pos;
        float s = -INFINITY;
        const size_t row = valid ? key_row(p, table, key, kvh) : 0;  // (0: a row of the reserved page, read for nothing)
        // the values of the tile's first keys are requested before the scores need its keys: one trip to memory, not two
        float v[BATCH][VE];
        auto values_from = [&](int j0) {
#pragma unroll
          for (int j = 0; j < BATCH; ++j) {
            const float* from = p.pages + __shfl_sync(0xffffffffu, (unsigned long long)row, j0 + j) + values;
#pragma unroll
            for (int e = 0; e < VE; ++e) v[j][e] = lane + 32 * e < d ? from[lane + 32 * e] : 0.f;
          }
        };
        values_from(0);
        if (valid) {
          float dot = 0.f;
#pragma unroll
          for (int base = 0; base < DP; base += 64) {  // a key's 256 bytes are requested at once
            float4 k[16];
#pragma unroll
            for (int c = 0; c < 16; ++c)
              k[c] = base + 4 * c < d ? *reinterpret_cast<const float4*>(p.pages + row + base + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const float4 qv = *reinterpret_cast<const float4*>(my_q + base + 4 * c);
              dot = fmaf(qv.x, k[c].x, dot);
              dot = fmaf(qv.y, k[c].y, dot);
              dot = fmaf(qv.z, k[c].z, dot);
              dot = fmaf(qv.w, k[c].w, dot);
            }
          }
          s = scored(dot, p.scale, p.softcap);
        }
        const float top = warp_max(s), w = part.weight(s, top, valid);
        part.rescale(top, warp_sum(w));
        const int begin = lo > start ? lo - start : 0, end = pos - start < 31 ? pos - start : 31;
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += BATCH) {
          if (j0 > end) break;
          if (j0) values_from(j0);
#pragma unroll
          for (int j = 0; j < BATCH; ++j) {
            const float wj = __shfl_sync(0xffffffffu, w, j0 + j);
            if (j0 + j >= begin && j0 + j <= end) {
#pragma unroll
              for (int e = 0; e < VE; ++e) part.acc[e] = fmaf(wj, v[j][e], part.acc[e]);
            }
          }
        }
      }
#pragma unroll
      for (int e = 0; e < VE; ++e) parts[buf][warp][lane + 32 * e] = part.acc[e];
      if (lane == 0) {
        parts[buf][warp][DP] = part.m;
        parts[buf][warp][DP + 1] = part.l;
      }
    }
    __syncthreads();  // (the round after the next overwrites this buffer, behind another barrier)
    if (heads == 1 && i < DP)
      for (int w = 0; w < SINGLE_WARPS && first + w <= pos / CHUNK_KEYS; ++w) {
        const float acc[1] = {parts[buf][w][i]};
        total.merge(parts[buf][w][DP], parts[buf][w][DP + 1], acc);
      }
  }
  if (heads == 1) {
    if (i < DP) write_out(p, t, h0, i, total.acc[0], 1.f / total.l);
    return;
  }
  for (int e = threadIdx.x; e < heads * DP; e += SINGLE_WARPS * 32) {
    const int head = h0 + e / DP;
    if (head >= p.nh) continue;
    total = nothing_yet(head);
    for (int w = 0; w < chunks; ++w) {
      const float* part = parts[0][e / DP * per + w];
      const float acc[1] = {part[e % DP]};
      total.merge(part[DP], part[DP + 1], acc);
    }
    write_out(p, t, head, e % DP, total.acc[0], 1.f / total.l);
  }
}

// Bound by shared-memory reads and the softmax's shuffles; the tile's keys and values, one 16-byte read a lane instead of a row
// of its own in global memory, serve 32 packed rows.  509 tokens, 14 heads of 64: 87 us (one warp a (token, head): 308 us);
// with four rows a warp and eight warps 89 us, and 10 % more beside other requests.
constexpr int ROWS_WARPS = 16, ROWS_A_WARP = 2, PACKED = ROWS_WARPS * ROWS_A_WARP;
template <int DP> constexpr int ROWS_SMEM = (PACKED * DP + 32 * (DP + 4) + 32 * DP + PACKED * 32) * 4;

// A block takes PACKED / group consecutive tokens at one KV head; row r is token r / group, head r % group of the group.  The
// tokens may belong to several requests: gridDim.z blocks take them in turn (requests one after the other in a block: 32 of 5
// tokens at 28 heads of 128, KV heads of 7, 23 us, side by side 15.7).
template <int DP>
__global__ void __launch_bounds__(ROWS_WARPS * 32, DP == 64 ? 2 : 1) attention_f32_rows_kernel(const ChunkArgs p) {
  tl::pdl_wait();
  tl::pdl_launch_dependents();
  constexpr int VE = DP / 32, NT = ROWS_WARPS * 32, COPIES = 32 * DP / 4 / NT, R = ROWS_A_WARP;
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                       // [PACKED][DP]
  float* ks = qs + PACKED * DP;           // [32][DP + 4]
  float* vs = ks + 32 * (DP + 4);         // [32][DP]
  float* ws = vs + 32 * DP;               // [PACKED][32] weights
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, d = p.d;
  const int group = p.nh / p.nkv, span = PACKED / group;
  const int kvh = blockIdx.y, t0 = (int)(gridDim.x - 1 - blockIdx.x) * span;  // the last tokens see the most keys: first
  const int count = p.tokens - t0 < span ? p.tokens - t0 : span;
  const size_t values = (size_t)p.nkv * p.page_size * d;
  const int my_req = lane < count ? p.token_req[t0 + lane] : 0, my_pos = lane < count ? p.positions[t0 + lane] : 0;  // (span <= 32)
  bool queries_here = false;
  const int few = few_tokens(group);
  for (int a = 0, b, turn = 0; a < count; a = b) {  // tokens [a, b) of one request
    const int req = __shfl_sync(0xffffffffu, my_req, a);
    const unsigned others = ~__ballot_sync(0xffffffffu, lane < count && my_req == req) >> a;
    b = others ? a + __ffs(others) - 1 : count;
    // the other kernel's (the run may go on in the blocks beside this one)
    const bool all_here = (a > 0 || t0 == 0) && (b < count || t0 + count == p.tokens);
    if (b - a <= few && (all_here || among_few(p, t0 + a, few))) continue;
    if (turn++ % gridDim.z != blockIdx.z) continue;  // another block's
    const bool here = lane >= a && lane < b;
    const int least = __reduce_min_sync(0xffffffffu, here ? first_key(my_pos, p.window) : INT_MAX);
    const int most = __reduce_max_sync(0xffffffffu, here ? my_pos : -1);
    if (!queries_here) {  // (read behind the first tile's barriers)
      for (int e = tid; e < PACKED * DP; e += NT) {
        const int r = e / DP, i = e % DP, token = r / group;
        qs[e] = (token < count && i < d) ? p.q[(size_t)(t0 + token) * p.q_stride + (size_t)(kvh * group + r % group) * d + i] : 0.f;
      }
      queries_here = true;
    }
    const int* table = p.block_table + (size_t)req * p.table_width;
    float4 kr[COPIES], vr[COPIES];
    auto fetch = [&](int start) {
#pragma unroll
      for (int c = 0; c < COPIES; ++c) {
        const int e = tid + c * NT, j = e / (DP / 4), i = e % (DP / 4) * 4;
        kr[c] = vr[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (start + j >= least && start + j <= most && i < d) {
          const float* k = p.pages + key_row(p, table, start + j, kvh) + i;
          kr[c] = *reinterpret_cast<const float4*>(k);
          vr[c] = *reinterpret_cast<const float4*>(k + values);
        }
      }
    };
    int pos[R], lo[R];
    bool live[R], seen[R];
    Softmax<VE> total[R], part[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = warp * R + r, token = row / group;
      live[r] = row < span * group && token >= a && token < b;
      pos[r] = __shfl_sync(0xffffffffu, my_pos, token & 31);
      if (!live[r]) pos[r] = -1;
      lo[r] = live[r] ? first_key(pos[r], p.window) : 0;
      seen[r] = false;
      total[r].clear();
      part[r].clear();
      if (p.sink) {
        total[r].m = p.sink_values && live[r] ? p.sink_values[kvh * group + row % group] : 0.f;
        total[r].l = 1.f;
      }
    }
    const int start0 = least & ~31;
    fetch(start0);
    for (int start = start0; start <= most; start += 32) {
      __syncthreads();  // the tile before has been read
#pragma unroll
      for (int c = 0; c < COPIES; ++c) {
        const int e = tid + c * NT, j = e / (DP / 4), i = e % (DP / 4) * 4;
        *reinterpret_cast<float4*>(ks + j * (DP + 4) + i) = kr[c];
        *reinterpret_cast<float4*>(vs + j * DP + i) = vr[c];
      }
      __syncthreads();
      if (start + 32 <= most) fetch(start + 32);
      unsigned mask[R], any = 0, all = 0xffffffffu;
      const int key = start + lane;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        mask[r] = __ballot_sync(0xffffffffu, key >= lo[r] && key <= pos[r]);
        any |= mask[r];
        all &= mask[r];
      }
      if (any) {
        float dot[R];
#pragma unroll
        for (int r = 0; r < R; ++r) dot[r] = 0.f;
#pragma unroll 4
        for (int c = 0; c < d; c += 4) {
          const float4 k = *reinterpret_cast<const float4*>(ks + lane * (DP + 4) + c);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float4 qv = *reinterpret_cast<const float4*>(qs + (warp * R + r) * DP + c);
            dot[r] = fmaf(qv.x, k.x, dot[r]);
            dot[r] = fmaf(qv.y, k.y, dot[r]);
            dot[r] = fmaf(qv.z, k.z, dot[r]);
            dot[r] = fmaf(qv.w, k.w, dot[r]);
          }
        }
        // the rows' maxima and sums together: their shuffles overlap
        float score[R], top[R], weight[R], sum[R];
#pragma unroll
        for (int r = 0; r < R; ++r) top[r] = score[r] = mask[r] >> lane & 1 ? scored(dot[r], p.scale, p.softcap) : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int r = 0; r < R; ++r) top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], o));
#pragma unroll
        for (int r = 0; r < R; ++r) sum[r] = weight[r] = part[r].weight(score[r], top[r], mask[r] >> lane & 1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int r = 0; r < R; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (mask[r]) part[r].rescale(top[r], sum[r]);
          seen[r] |= mask[r] != 0;
          ws[(warp * R + r) * 32 + lane] = weight[r];
        }
        __syncwarp();
#pragma unroll 2
        for (int j = 0; j < 32; j += 4) {
          if (start + j > most) break;
          float4 w[R];
#pragma unroll
          for (int r = 0; r < R; ++r) w[r] = *reinterpret_cast<const float4*>(ws + (warp * R + r) * 32 + j);
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            float v[VE];
#pragma unroll
            for (int e = 0; e < VE; ++e) v[e] = vs[(j + jj) * DP + lane + 32 * e];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const float wj = jj == 0 ? w[r].x : (jj == 1 ? w[r].y : (jj == 2 ? w[r].z : w[r].w));
              // a key that the row does not see adds nothing, whatever its value row holds
              if (all == 0xffffffffu || mask[r] >> (j + jj) & 1) {
#pragma unroll
                for (int e = 0; e < VE; ++e) part[r].acc[e] = fmaf(wj, v[e], part[r].acc[e]);
              }
            }
          }
        }
        __syncwarp();  // the weights have been read
      }
      if ((start + 32) % CHUNK_KEYS == 0 || start + 32 > most) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (seen[r]) {
            total[r].merge(part[r].m, part[r].l, part[r].acc);
            part[r].clear();
            seen[r] = false;
          }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (live[r]) {
        const int row = warp * R + r;
        const float inv = 1.f / total[r].l;
#pragma unroll
        for (int e = 0; e < VE; ++e) write_out(p, t0 + row / group, kvh * group + row % group, lane + 32 * e, total[r].acc[e], inv);
      }
    __syncthreads();  // (the next request's first tile)
  }
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

// The layers whose 32-bit rows go by chunks.  Nothing here depends on the step.
bool in_chunks(int nh, int nkv, int d, int keep, int chunks) {
  return d <= 128 && d % 4 == 0 && nh / nkv <= PACKED && keep == 0 && chunks == 1 && nkv <= 65535;
}

// ``portions`` requests bring more than one token; none brings fewer than ``least`` or more than ``most``; those of up to 8 lie in
// the first few_rows rows.
template <int DP>
int launch_chunks(ChunkArgs p, int portions, int least, int most, int few_rows, cudaStream_t stream) {
  const int group = p.nh / p.nkv, span = PACKED / group, few = few_tokens(group);
  p.all_few = most <= few;
  if (p.all_few) few_rows = p.tokens;
  else if (least > few) few_rows = 0;
  if (!p.all_few) {
    static bool configured = false;
    if (!configured && ROWS_SMEM<DP> > 48 * 1024) {
      const cudaError_t err = cudaFuncSetAttribute(attention_f32_rows_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM<DP>);
      if (err != cudaSuccess) return (int)err;
      configured = true;
    }
    // as many blocks for the same tokens as there are requests among them, up to four
    const int turns = (int)min(4ll, 1 + ((long long)span * portions + p.tokens / 2) / p.tokens);
    tl::launch_kernel(attention_f32_rows_kernel<DP>, dim3((p.tokens + span - 1) / span, p.nkv, turns), ROWS_WARPS * 32, ROWS_SMEM<DP>, stream, p);
    const int rc = TL_LAUNCH_CHECK();
    if (rc || few_rows == 0) return rc;
  }
  const unsigned blocks = (unsigned)few_rows * p.nh;
  if (blocks > 4u * sm_count())
    tl::launch_kernel(attention_f32_single_kernel<DP, true>, dim3(blocks), SINGLE_WARPS * 32, 0, stream, p);
  else
    tl::launch_kernel(attention_f32_single_kernel<DP, false>, dim3(blocks), SINGLE_WARPS * 32, 0, stream, p);
  const int rc = TL_LAUNCH_CHECK();
  return rc || p.all_few ? rc : -2;  // two kernels
}

}  // namespace

TL_DEBUG_READER(tl_attention_generic_debug_error)

// Hints about the step (1, 1, ``tokens`` and ``tokens`` where nothing is known): how many requests bring more than one token, the fewest and
// the most tokens that one brings, and the row behind the last of a request of up to 8 tokens.
// Returns 0, an error code, or -2 where two kernels were launched.
extern "C" int tl_attention_generic(const void* q, int q_stride, const void* pages, int dtype,
                                    const int* block_table, int table_width, const int* token_req,
                                    const int* positions, void* out, int out_stride, int tokens,
                                    int nh, int nkv, int d, int page_size, int window, float scale,
                                    int num_pages, float softcap, int sink, const float* sink_values,
                                    const float* gate, int gate_stride, int keep, int chunks, int v_cols, int portions, int least,
                                    int most, int few_rows,
                                    cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (d <= 0 || d > MAX_D || nkv <= 0 || nh % nkv || page_size <= 0) return TL_ERR_UNSUPPORTED;
  if (keep < 0 || (chunks != 1 && chunks != nkv) || v_cols <= 0 || v_cols > d) return TL_ERR_UNSUPPORTED;
  if (dtype == TL_DTYPE_F32 && in_chunks(nh, nkv, d, keep, chunks) && (reinterpret_cast<uintptr_t>(pages) & 15) == 0) {
    const ChunkArgs p{(const float*)q, (const float*)pages, block_table, token_req, positions, (float*)out, sink_values, gate,
                      q_stride, table_width, out_stride, tokens, nh, nkv, d, page_size, window, num_pages, sink, gate_stride,
                      v_cols, 0, scale, softcap};
    few_rows = few_rows < tokens ? few_rows : tokens;
    return d <= 64 ? launch_chunks<64>(p, portions, least, most, few_rows, stream)
                   : launch_chunks<128>(p, portions, least, most, few_rows, stream);
  }
  const size_t smem = (size_t)WARPS * chunks * d * sizeof(float);
  if (smem > 200 * 1024) return TL_ERR_UNSUPPORTED;
  if (smem > 48 * 1024) {
    const cudaError_t err = dtype == TL_DTYPE_F32
        ? cudaFuncSetAttribute(attention_generic_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
        : cudaFuncSetAttribute(attention_generic_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
  }
  const int wide = d % 8 == 0 && q_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(pages) & 31) == 0;
  const long long items = (long long)tokens * nh;
  const unsigned blocks = (unsigned)((items + WARPS - 1) / WARPS);
  if (dtype == TL_DTYPE_F32)
    tl::launch_kernel(attention_generic_kernel<float>, blocks, WARPS * 32, smem, stream,
        (const float*)q, q_stride, (const float*)pages, block_table, table_width, token_req,
        positions, (float*)out, out_stride, tokens, nh, nkv, d, page_size, window, scale, num_pages, softcap, sink,
        sink_values, gate, gate_stride, wide, keep, chunks, v_cols);
  else
    tl::launch_kernel(attention_generic_kernel<__nv_bfloat16>, blocks, WARPS * 32, smem, stream,
        (const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)pages, block_table, table_width,
        token_req, positions, (__nv_bfloat16*)out, out_stride, tokens, nh, nkv, d, page_size, window,
        scale, num_pages, softcap, sink, sink_values, gate, gate_stride, wide, keep, chunks, v_cols);
  return TL_LAUNCH_CHECK();
}
