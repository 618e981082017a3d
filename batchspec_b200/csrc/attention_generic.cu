// Paged causal attention, generic path: any head_dim up to 256, any number of heads and groups, any page size, float32 or
// bfloat16 storage, float32 arithmetic throughout.  A block holds R consecutive (query token, query head of the group) rows of
// one request and kv head.  Keys are visited in chunks of 32 that start at multiples of 32 of the key index; chunk c belongs to
// share c % W, which keeps a running softmax of its chunks for every row, and the shares' results are joined in their order at
// the end.  A share is a warp's; attn_row_kernel below has one warp per row, which takes the shares one after the other.  So the
// order of every sum depends only on the query's own position (and the head sizes, which choose W), not on how the request
// was cut into steps, on what else is in the batch or on which of the kernels runs: a key that a row does not see adds
// an exact nothing.
//
// Cache layer layout: [pages][k: [Hkv][page_size][hd] | v: [Hkv][page_size][vd]] (vd = hd unless values have a size
// of their own).
//
// Masks: causal; ``window`` > 0 keeps the last ``window`` keys; ``chunk`` > 0 keeps the keys of the query's own
// chunk, floor(key / chunk) == floor(query / chunk), chunks counted from position 0 of the request.  ``sink``: one
// float32 per query head: exp(sink) is added to the softmax denominator, nothing to the numerator.  ``softcap`` c > 0:
// a score s (after the scale) becomes c tanh(s / c).  ``v_is_k``: the values are the keys; a page then holds
// [Hkv][page_size][hd] only.  ``gate`` (float32 rows [Hq*vd] of stride gate_stride, or null): the output is multiplied
// element by element by sigmoid(gate); ``out_scale`` multiplies it too; output rows have stride out_stride.
//
// ``slopes`` (float32 per query head, or null): slope_h * (query - key) is taken off a token's score.  ``pool`` P > 0
// (with a window W): before the window a query also sees one entry per block of P tokens that lies wholly before it,
// floor((query - W + 1) / P) of them; they have pages and a table of their own (same page layout, entry b = block b)
// and take part in the same softmax, first.  ``pool`` < 0 (with a window): the request's first -pool tokens stay visible
// when the window has passed them; they are visited first, from the tokens' own pages.
#include "common.cuh"
#include <cuda_pipeline.h>
#include <math.h>
#include <type_traits>
using namespace bspec;

namespace {
constexpr int MAX_HD = 256;

// four consecutive numbers as float32
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&v.x), b = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
  return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
// four numbers of a key into shared memory: a copy that runs on its own, or through registers where the type changes
__device__ __forceinline__ void stage4(float* dst, const float* src) { __pipeline_memcpy_async(dst, src, 16); }
__device__ __forceinline__ void stage4(float* dst, const __nv_bfloat16* src) { *reinterpret_cast<float4*>(dst) = load4(src); }

// Heads of up to 32 ND numbers.  Bound by shared memory: a lane's key row lies in shared memory (32 rows padded by four
// floats), the R queries are broadcast, so 4 numbers of the head cost 1 + R loads of 16 bytes for 4 R multiply-adds; with
// the chunk's weights in shared memory the values' sum is the same.  The next chunk's keys are copied under the values'
// sum.  Measured in whole passes at the 1B sizes, 16 layers (32 heads of 64 over 8 kv heads): a decode step of 4 requests of
// 33 to 500 keys 10.15 -> 2.01 ms, prompts of 61, 207 and 700 tokens 97.0 -> 57.7 ms, against a warp per query row with a key
// per lane and nothing shared (536 us a layer in the decode step).
template <int ND> struct Shape { static constexpr int W = ND == 8 ? 4 : 8, LDK = 32 * ND + 4; };

constexpr int attn_smem(int nd, int r) {
  const int w = nd == 8 ? 4 : 8;
  return (w * 32 * (32 * nd + 4) + r * 32 * nd + w * r * 32 + 2 * w * r) * 4 + w * 32 * 16 + r * 8 * 2;
}

// One row's results, ``n`` shares in their order: part[w * part_step + d] with maximum and sum at ml[w * ml_step].  ``gp``: one
// gate logit per output number, or (gate_per_head) one per head.
template <typename T, int ND>
__device__ __forceinline__ void join_row(const float* part, int part_step, const float* ml, int ml_step, int n,
                                         const float* __restrict__ sink, T* __restrict__ op, int vd,
                                         const float* __restrict__ gp, int gate_per_head, float out_scale) {
  const int lane = threadIdx.x & 31;
  float top = sink != nullptr ? *sink : -INFINITY;
  for (int w = 0; w < n; ++w) top = fmaxf(top, ml[w * ml_step]);
  float sum = 0.f, o[ND];
#pragma unroll
  for (int i = 0; i < ND; ++i) o[i] = 0.f;
  for (int w = 0; w < n; ++w) {
    const float mw = ml[w * ml_step], lw = ml[w * ml_step + 1];
    if (mw == -INFINITY && lw == 0.f) continue;             // the share has no key for this row
    const float f = expf(mw - top);
    sum = fmaf(lw, f, sum);
#pragma unroll
    for (int i = 0; i < ND; ++i) o[i] = fmaf(part[(size_t)w * part_step + lane + 32 * i], f, o[i]);
  }
  if (sink != nullptr) sum += expf(*sink - top);            // one more term of the denominator only
  const float inv = 1.f / sum;
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    const int d = lane + 32 * i;
    if (d < vd) {
      float x = o[i] * inv;
      if (gp != nullptr) x = x / (1.f + expf(-gp[gate_per_head ? 0 : d]));
      op[d] = from_f32<T>(x * out_scale);
    }
  }
}

template <typename T, int ND, int R>
__global__ void __launch_bounds__(Shape<ND>::W * 32)
attn_generic_kernel(const T* __restrict__ q, long long q_row_stride, T* __restrict__ out,
                    const T* __restrict__ cache, const int* __restrict__ qo_indptr,
                    const int* __restrict__ positions, const int* __restrict__ kv_indptr,
                    const int* __restrict__ kv_indices, int Hq, int Hkv, int hd, int page_size, float scale,
                    int window, long long n_pages, int vd, int chunk, const float* __restrict__ sink,
                    float softcap, int v_is_k, const float* __restrict__ gate, long long gate_stride,
                    long long out_stride, float out_scale, int gate_per_head, const float* __restrict__ slopes,
                    int pool, const T* __restrict__ pool_cache, const int* __restrict__ pool_indptr,
                    const int* __restrict__ pool_indices, long long pool_pages) {
  bspec::pdl_prologue(7);
  constexpr int W = Shape<ND>::W, LDK = Shape<ND>::LDK, D = 32 * ND;
  constexpr int UK = R <= 4 && ND <= 4 ? 8 : 2;             // quads of values asked for at a time
  extern __shared__ __align__(16) float smem_f[];
  float* kbuf = smem_f;                                     // [W][32][LDK]
  float* qs = kbuf + W * 32 * LDK;                          // [R][D]
  float* ps = qs + R * D;                                   // [W][R][32]
  float* ml = ps + W * R * 32;                              // [W][R][2]: maximum, sum
  long long* offs = reinterpret_cast<long long*>(ml + 2 * W * R);     // [W][32][2]: where a key and its value lie, -1: nowhere
  int2* seen = reinterpret_cast<int2*>(offs + W * 64);      // [2][R]: first and last key that a row sees; of the second source
  const int e = blockIdx.y, kvh = blockIdx.z, G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_begin = qo_indptr[e], rows = (qo_indptr[e + 1] - q_begin) * G;
  const int row0 = (int)(gridDim.x - 1 - blockIdx.x) * R;   // the tiles with the most keys first
  if (row0 >= rows) return;
  const int nr = min(R, rows - row0);
  for (int i = threadIdx.x; i < R * (D / 4); i += W * 32) {
    const int r = i / (D / 4), d = i % (D / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < nr && d < hd) {
      const T* qp = q + (size_t)(q_begin + (row0 + r) / G) * q_row_stride + (size_t)(kvh * G + (row0 + r) % G) * hd + d;
      v = make_float4(to_f32(qp[0]), d + 1 < hd ? to_f32(qp[1]) : 0.f, d + 2 < hd ? to_f32(qp[2]) : 0.f, d + 3 < hd ? to_f32(qp[3]) : 0.f);
    }
    *reinterpret_cast<float4*>(qs + r * D + d) = v;
  }
  if (threadIdx.x < R) {
    int2 own = make_int2(0, -1), other = make_int2(0, -1);
    if ((int)threadIdx.x < nr) {
      const int pos = positions[q_begin + (row0 + threadIdx.x) / G];
      own = make_int2(window > 0 ? max(0, pos - window + 1) : 0, pos);
      if (chunk > 0) own.x = max(own.x, (pos / chunk) * chunk);
      if (pool != 0) other.y = bspec::pooled_seen(pos, window, pool) - 1;
    }
    seen[threadIdx.x] = own;
    seen[R + threadIdx.x] = other;
  }
  __syncthreads();

  const size_t k_elems = (size_t)Hkv * page_size * hd;      // the keys of a page; its values follow them
  const size_t page_elems = k_elems + (v_is_k ? (size_t)0 : (size_t)Hkv * page_size * vd);
  float* kb = kbuf + warp * 32 * LDK;
  float* pw = ps + warp * R * 32;
  long long* off = offs + warp * 64;
  const int quads = (hd + 3) / 4;
  float acc[R][ND], m[R], l[R];                             // l: this lane's keys only
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int i = 0; i < ND; ++i) acc[r][i] = 0.f;
  }

  // all chunks of one source (the request's tokens, or what it sees before the window) that fall to this warp
  auto visit = [&](const int2* rng, const int* tab, const T* base, long long pages, bool biased) {
    int lo = 1 << 30, hi = -1;
    for (int r = 0; r < nr; ++r)
      if (rng[r].y >= rng[r].x) { lo = min(lo, rng[r].x); hi = max(hi, rng[r].y); }
    if (hi < 0) return;
    const bool vec = ((hd | (int)page_elems) & 3) == 0 && ((uintptr_t)base & (4 * sizeof(T) - 1)) == 0;     // keys start on whole quads
    auto fetch = [&](int c) {
      const int key = 32 * c + lane;
      bool valid = key >= lo && key <= hi;
      if (valid && !bspec::in_range(tab[key / page_size], pages, 107)) valid = false;
      long long ko = -1, vo = -1;
      if (valid) {
        const size_t page = (size_t)tab[key / page_size] * page_elems;
        const size_t row = (size_t)kvh * page_size + (size_t)(key % page_size);
        ko = (long long)(page + row * hd);
        vo = v_is_k ? ko : (long long)(page + k_elems + row * vd);
      }
      off[2 * lane] = ko;
      off[2 * lane + 1] = vo;
      __syncwarp();
      if (vec) {
        for (int i = lane; i < 32 * quads; i += 32) {
          const int row = i / quads, d = (i - row * quads) * 4;
          const long long at = off[2 * row];
          if (at >= 0) stage4(kb + row * LDK + d, base + at + d);
        }
      } else {
        for (int i = lane; i < 128 * quads; i += 32) {
          const int row = i / (4 * quads), d = i - row * 4 * quads;
          const long long at = off[2 * row];
          kb[row * LDK + d] = at >= 0 && d < hd ? to_f32(base[at + d]) : 0.f;
        }
      }
      __pipeline_commit();
    };
    const int c_last = hi / 32;
    int c = lo / 32 + (warp + W - lo / 32 % W) % W;          // the first chunk from lo / 32 on with c % W == warp
    if (c <= c_last) fetch(c);
    for (; c <= c_last; c += W) {
      __pipeline_wait_prior(0);
      __syncwarp();
      const int key = 32 * c + lane;
      const bool valid = off[2 * lane] >= 0;
      float s[R];
#pragma unroll
      for (int r = 0; r < R; ++r) s[r] = 0.f;
      for (int d = 0; d < hd; d += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(kb + lane * LDK + d);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 q4 = *reinterpret_cast<const float4*>(qs + r * D + d);
          s[r] = fmaf(q4.x, k4.x, s[r]);
          s[r] = fmaf(q4.y, k4.y, s[r]);
          s[r] = fmaf(q4.z, k4.z, s[r]);
          s[r] = fmaf(q4.w, k4.w, s[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int2 see = rng[r];
        const bool on = valid && key >= see.x && key <= see.y;
        float x = -INFINITY;
        if (on) {
          x = s[r] * scale;
          if (softcap > 0.f) x = softcap * tanhf(x / softcap);
          // one rounding, fused by name so that every instance has the same bits
          if (biased) x = __fmaf_rn(-slopes[kvh * G + (row0 + r) % G], (float)(seen[r].y - key), x);
        }
        const float top = fmaxf(m[r], warp_max(x));
        const float p = x == -INFINITY ? 0.f : expf(x - top);             // (unseen, or a score of -inf in a chunk of nothing else)
        const float corr = m[r] == top ? 1.f : expf(m[r] - top);          // (also where the row sees nothing yet)
        l[r] = fmaf(l[r], corr, p);
        if (corr != 1.f) {
#pragma unroll
          for (int i = 0; i < ND; ++i) acc[r][i] *= corr;
        }
        m[r] = top;
        pw[r * 32 + lane] = p;
      }
      // the values' places, before the next chunk's take theirs
      const long long mine = off[2 * lane + 1];
      __syncwarp();
      if (c + W <= c_last) fetch(c + W);
#pragma unroll UK
      for (int k4 = 0; k4 < 32; k4 += 4) {
        float v[4][ND];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const long long at = __shfl_sync(0xffffffffu, mine, k4 + u);
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            const int d = lane + 32 * i;
            v[u][i] = at >= 0 && d < vd ? to_f32(base[at + d]) : 0.f;
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 p4 = *reinterpret_cast<const float4*>(pw + r * 32 + k4);
          const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (p[u] != 0.f) {                              // an unseen key's value may be anything
#pragma unroll
              for (int i = 0; i < ND; ++i) acc[r][i] = fmaf(p[u], v[u][i], acc[r][i]);
            }
        }
      }
      __syncwarp();
    }
  };
  const int* table = kv_indices + kv_indptr[e];
  if (pool < 0) visit(seen + R, table, cache, n_pages, slopes != nullptr);
  if (pool > 0) visit(seen + R, pool_indices + pool_indptr[e], pool_cache, pool_pages, false);
  visit(seen, table, cache, n_pages, slopes != nullptr);

  // join the warps in their order
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float sum = warp_sum(l[r]);
    if (lane == 0) {
      ml[(warp * R + r) * 2] = m[r];
      ml[(warp * R + r) * 2 + 1] = sum;
    }
  }
  __syncthreads();                                          // and every warp is done with its keys
  float* part = smem_f;                                     // [W][R][D]: where the keys were
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < ND; ++i) part[(size_t)(warp * R + r) * D + lane + 32 * i] = acc[r][i];
  __syncthreads();
  for (int r = warp; r < nr; r += W) {
    const int t = q_begin + (row0 + r) / G, h = kvh * G + (row0 + r) % G;
    join_row<T, ND>(part + (size_t)r * D, R * D, ml + 2 * r, 2 * R, W, sink != nullptr ? sink + h : nullptr,
                    out + (size_t)t * out_stride + (size_t)h * vd, vd,
                    gate != nullptr ? gate + (size_t)t * gate_stride + (size_t)h * (gate_per_head ? 1 : vd) : nullptr, gate_per_head,
                    out_scale);
  }
}

// The same shares for portions of several tokens, laid out for the multiply-adds: a lane takes 4 keys x R / 4 rows of a chunk's
// scores (keys lane % 8 + 8 j, rows lane / 8 + 4 i, which keeps the order in which a row's weights are added up), then R / 4 rows
// x ND quads of the values' sum, so 16 bytes of shared memory serve 8 to 16 multiply-adds where the layout above has 4, a row's maximum
// takes three shuffles, and the values come through shared memory as quads: they take the place of the chunk's keys once the scores
// are there.  128 registers keep two blocks of eight warps on an SM where the 168 of the layout above kept one.  Measured at the 1B
// sizes in float32 (32 heads of 64 over 8 kv heads, prompts of 61, 207 and 700 tokens): 371 -> 169 us a layer, the pass 22.25 ->
// 18.95 ms.  Bound by the multiply-adds, the exponentials and the latency of a chunk's two copies: a warp has at most three chunks
// there.  Other sizes, us, layout above / this one: float32, 24/8 x 128 the same prompts 393 / 255, 64 tokens beside 63 decoded ones of
// 2,000 keys 877 / 444, 16/4 x 256 861 / 551 and 1,384 / 504; bfloat16, whose values this one has to convert on their way, 32/8 x 64
// 381 / 204, 24/8 x 128 488 / 415, 12/2 x 80 213 / 160, but 16/4 x 256 1,197 / 1,218 and 8/8 x 256, 16 tokens beside 7 decoded ones,
// 283 / 296: bfloat16 heads above 128 numbers keep the layout above.  So do decoded tokens: their rows are few, and the next keys
// come under the values' sum.
constexpr int LDP = 40;                                     // a row of weights: four rows of a quad lie in different banks

constexpr int attn_tile_smem(int nd, int r) {
  const int w = nd == 8 ? 4 : 8;
  return (w * 32 * (32 * nd + 4) + r * (32 * nd + 4) + w * r * LDP + 2 * w * r) * 4 + w * 32 * 16 + r * 8 * 2;
}

template <typename T, int ND, int R>
__global__ void __launch_bounds__(Shape<ND>::W * 32, ND == 2 ? 2 : 1)
attn_tile_kernel(const T* __restrict__ q, long long q_row_stride, T* __restrict__ out,
                 const T* __restrict__ cache, const int* __restrict__ qo_indptr,
                 const int* __restrict__ positions, const int* __restrict__ kv_indptr,
                 const int* __restrict__ kv_indices, int Hq, int Hkv, int hd, int page_size, float scale,
                 int window, long long n_pages, int vd, int chunk, const float* __restrict__ sink,
                 float softcap, int v_is_k, const float* __restrict__ gate, long long gate_stride,
                 long long out_stride, float out_scale, int gate_per_head, const float* __restrict__ slopes,
                 int pool, const T* __restrict__ pool_cache, const int* __restrict__ pool_indptr,
                 const int* __restrict__ pool_indices, long long pool_pages) {
  bspec::pdl_prologue(7);
  constexpr int W = Shape<ND>::W, LDK = Shape<ND>::LDK, D = 32 * ND, LDQ = D + 4, NR = R / 4;
  extern __shared__ __align__(16) float smem_f[];
  float* kbuf = smem_f;                                     // [W][32][LDK] a chunk's keys, then its values
  float* qs = kbuf + W * 32 * LDK;                          // [R][LDQ]
  float* ps = qs + R * LDQ;                                 // [W][R][LDP]
  float* ml = ps + W * R * LDP;                             // [W][R][2]: maximum, sum
  long long* offs = reinterpret_cast<long long*>(ml + 2 * W * R);     // [W][32][2]: where a key and its value lie, -1: nowhere
  int2* seen = reinterpret_cast<int2*>(offs + W * 64);      // [2][R]: first and last key that a row sees; of the second source
  const int e = blockIdx.y, kvh = blockIdx.z, G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kg = lane & 7, rg = lane >> 3;
  const int q_begin = qo_indptr[e], rows = (qo_indptr[e + 1] - q_begin) * G;
  const int row0 = (int)(gridDim.x - 1 - blockIdx.x) * R;   // the tiles with the most keys first
  if (row0 >= rows) return;
  const int nr = min(R, rows - row0);
  for (int i = threadIdx.x; i < R * (D / 4); i += W * 32) {
    const int r = i / (D / 4), d = i % (D / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < nr && d < hd) {
      const T* qp = q + (size_t)(q_begin + (row0 + r) / G) * q_row_stride + (size_t)(kvh * G + (row0 + r) % G) * hd + d;
      v = make_float4(to_f32(qp[0]), d + 1 < hd ? to_f32(qp[1]) : 0.f, d + 2 < hd ? to_f32(qp[2]) : 0.f, d + 3 < hd ? to_f32(qp[3]) : 0.f);
    }
    *reinterpret_cast<float4*>(qs + r * LDQ + d) = v;
  }
  if (threadIdx.x < R) {
    int2 own = make_int2(0, -1), other = make_int2(0, -1);
    if ((int)threadIdx.x < nr) {
      const int pos = positions[q_begin + (row0 + threadIdx.x) / G];
      own = make_int2(window > 0 ? max(0, pos - window + 1) : 0, pos);
      if (chunk > 0) own.x = max(own.x, (pos / chunk) * chunk);
      if (pool != 0) other.y = bspec::pooled_seen(pos, window, pool) - 1;
    }
    seen[threadIdx.x] = own;
    seen[R + threadIdx.x] = other;
  }
  __syncthreads();

  const size_t k_elems = (size_t)Hkv * page_size * hd;      // the keys of a page; its values follow them
  const size_t page_elems = k_elems + (v_is_k ? (size_t)0 : (size_t)Hkv * page_size * vd);
  float* kb = kbuf + warp * 32 * LDK;
  float* pw = ps + warp * R * LDP;
  long long* off = offs + warp * 64;
  float4 acc[NR][ND];
  float m[NR], l[NR][4];                                    // l: this lane's keys only
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    m[i] = -INFINITY;
#pragma unroll
    for (int j = 0; j < 4; ++j) l[i][j] = 0.f;
#pragma unroll
    for (int c = 0; c < ND; ++c) acc[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  // all chunks of one source (the request's tokens, or what it sees before the window) that fall to this warp
  auto visit = [&](const int2* rng, const int* tab, const T* base, long long pages, bool biased) {
    int lo = 1 << 30, hi = -1;
    for (int r = 0; r < nr; ++r)
      if (rng[r].y >= rng[r].x) { lo = min(lo, rng[r].x); hi = max(hi, rng[r].y); }
    if (hi < 0) return;
    const bool whole = ((uintptr_t)base & (4 * sizeof(T) - 1)) == 0;
    const bool vec[2] = {whole && ((hd | (int)page_elems) & 3) == 0, whole && ((hd | vd | (int)page_elems) & 3) == 0};     // whole quads
    auto stage = [&](int which, int n) {                    // the chunk's keys (0) or values (1), ``n`` numbers each
      if (vec[which]) {
        const int quads = n / 4, rows_on = 32 / quads, quads_on = 32 - rows_on * quads;
        for (int row = lane / quads, d = lane % quads; row < 32;) {
          const long long at = off[2 * row + which];
          if (at >= 0) stage4(kb + row * LDK + 4 * d, base + at + 4 * d);
          row += rows_on;
          if ((d += quads_on) >= quads) d -= quads, ++row;
        }
      } else {
        const int wide = (n + 3) / 4 * 4;
        for (int i = lane; i < 32 * wide; i += 32) {
          const int row = i / wide, d = i - row * wide;
          const long long at = off[2 * row + which];
          kb[row * LDK + d] = at >= 0 && d < n ? to_f32(base[at + d]) : 0.f;
        }
      }
      __pipeline_commit();
    };
    auto fetch = [&](int c) {
      const int key = 32 * c + lane;
      bool valid = key >= lo && key <= hi;
      if (valid && !bspec::in_range(tab[key / page_size], pages, 107)) valid = false;
      long long ko = -1, vo = -1;
      if (valid) {
        const size_t page = (size_t)tab[key / page_size] * page_elems;
        const size_t row = (size_t)kvh * page_size + (size_t)(key % page_size);
        ko = (long long)(page + row * hd);
        vo = v_is_k ? ko : (long long)(page + k_elems + row * vd);
      }
      off[2 * lane] = ko;
      off[2 * lane + 1] = vo;
      __syncwarp();
      stage(0, hd);
    };
    const int c_last = hi / 32;
    int c = lo / 32 + (warp + W - lo / 32 % W) % W;          // the first chunk from lo / 32 on with c % W == warp
    if (c <= c_last) fetch(c);
    for (; c <= c_last; c += W) {
      __pipeline_wait_prior(0);
      __syncwarp();
      float s[NR][4];
#pragma unroll
      for (int i = 0; i < NR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
      for (int d = 0; d < hd; d += 4) {
        float4 k4[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) k4[j] = *reinterpret_cast<const float4*>(kb + (kg + 8 * j) * LDK + d);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const float4 q4 = *reinterpret_cast<const float4*>(qs + (rg + 4 * i) * LDQ + d);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            s[i][j] = fmaf(q4.x, k4[j].x, s[i][j]);
            s[i][j] = fmaf(q4.y, k4[j].y, s[i][j]);
            s[i][j] = fmaf(q4.z, k4[j].z, s[i][j]);
            s[i][j] = fmaf(q4.w, k4[j].w, s[i][j]);
          }
        }
      }
      bool valid[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) valid[j] = off[2 * (kg + 8 * j)] >= 0;
      __syncwarp();
      if (!v_is_k) stage(1, vd);                            // over the keys, under the softmax
      bool none = false;                                    // a weight is zero
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int r = rg + 4 * i;
        const int2 see = rng[r];
        float x[4], top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = 32 * c + kg + 8 * j;
          x[j] = -INFINITY;
          if (valid[j] && key >= see.x && key <= see.y) {
            x[j] = s[i][j] * scale;
            if (softcap > 0.f) x[j] = softcap * tanhf(x[j] / softcap);
            if (biased) x[j] = __fmaf_rn(-slopes[kvh * G + (row0 + r) % G], (float)(seen[r].y - key), x[j]);
          }
          top = fmaxf(top, x[j]);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        top = fmaxf(m[i], top);
        const float corr = m[i] == top ? 1.f : expf(m[i] - top);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = x[j] == -INFINITY ? 0.f : expf(x[j] - top);
          l[i][j] = fmaf(l[i][j], corr, p);
          none |= p == 0.f;
          pw[r * LDP + kg + 8 * j] = p;
        }
        if (corr != 1.f) {
#pragma unroll
          for (int b = 0; b < ND; ++b) acc[i][b].x *= corr, acc[i][b].y *= corr, acc[i][b].z *= corr, acc[i][b].w *= corr;
        }
        m[i] = top;
      }
      none = __any_sync(0xffffffffu, none);
      __pipeline_wait_prior(0);
      __syncwarp();
      auto sum = [&](auto guarded) {
#pragma unroll 2
        for (int k4 = 0; k4 < 32; k4 += 4) {
          float p[NR][4];
#pragma unroll
          for (int i = 0; i < NR; ++i) {
            const float4 p4 = *reinterpret_cast<const float4*>(pw + (rg + 4 * i) * LDP + k4);
            p[i][0] = p4.x, p[i][1] = p4.y, p[i][2] = p4.z, p[i][3] = p4.w;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int b = 0; b < ND; ++b) {
              const float4 v = *reinterpret_cast<const float4*>(kb + (k4 + u) * LDK + 32 * b + 4 * kg);
#pragma unroll
              for (int i = 0; i < NR; ++i)
                if (!decltype(guarded)::value || p[i][u] != 0.f) {     // an unseen key's value may be anything
                  acc[i][b].x = fmaf(p[i][u], v.x, acc[i][b].x);
                  acc[i][b].y = fmaf(p[i][u], v.y, acc[i][b].y);
                  acc[i][b].z = fmaf(p[i][u], v.z, acc[i][b].z);
                  acc[i][b].w = fmaf(p[i][u], v.w, acc[i][b].w);
                }
            }
        }
      };
      if (none) sum(std::true_type());
      else sum(std::false_type());
      __syncwarp();
      if (c + W <= c_last) fetch(c + W);
    }
  };
  const int* table = kv_indices + kv_indptr[e];
  if (pool < 0) visit(seen + R, table, cache, n_pages, slopes != nullptr);
  if (pool > 0) visit(seen + R, pool_indices + pool_indptr[e], pool_cache, pool_pages, false);
  visit(seen, table, cache, n_pages, slopes != nullptr);

  // join the warps in their order; a row's 32 sums of weights as warp_sum adds them
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    float sum = (l[i][0] + l[i][2]) + (l[i][1] + l[i][3]);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (kg == 0) {
      ml[(warp * R + rg + 4 * i) * 2] = m[i];
      ml[(warp * R + rg + 4 * i) * 2 + 1] = sum;
    }
  }
  __syncthreads();                                          // and every warp is done with its keys
  float* part = smem_f;                                     // [W][R][D]: where the keys were
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int b = 0; b < ND; ++b) *reinterpret_cast<float4*>(part + (size_t)(warp * R + rg + 4 * i) * D + 32 * b + 4 * kg) = acc[i][b];
  __syncthreads();
  for (int r = warp; r < nr; r += W) {
    const int t = q_begin + (row0 + r) / G, h = kvh * G + (row0 + r) % G;
    join_row<T, ND>(part + (size_t)r * D, R * D, ml + 2 * r, 2 * R, W, sink != nullptr ? sink + h : nullptr,
                    out + (size_t)t * out_stride + (size_t)h * vd, vd,
                    gate != nullptr ? gate + (size_t)t * gate_stride + (size_t)h * (gate_per_head ? 1 : vd) : nullptr, gate_per_head,
                    out_scale);
  }
}

// One warp per (query token, query head) row, for short requests and for many rows with keys of their own (by_rows):
// nothing is shared or staged, a lane reads its key itself, so a block needs a few KB instead of the 70 to 140 that keep one to
// three blocks on an SM above, and little code.  A warp takes the shares of the chunks one after the other, each from an empty
// softmax, and joins them as the kernel above does: a row has the same bits in both.
constexpr int ROW_WARPS = 4;

constexpr int attn_row_smem(int nd, int warps) { return warps * (32 * nd + (nd == 8 ? 4 : 8) * (32 * nd + 2)) * 4; }

template <typename T, int ND>
__global__ void __launch_bounds__(ROW_WARPS * 32)
attn_row_kernel(const T* __restrict__ q, long long q_row_stride, T* __restrict__ out,
                const T* __restrict__ cache, const int* __restrict__ qo_indptr,
                const int* __restrict__ positions, const int* __restrict__ kv_indptr,
                const int* __restrict__ kv_indices, int Hq, int Hkv, int hd, int page_size, float scale,
                int window, long long n_pages, int vd, int chunk, const float* __restrict__ sink,
                float softcap, int v_is_k, const float* __restrict__ gate, long long gate_stride,
                long long out_stride, float out_scale, int gate_per_head, const float* __restrict__ slopes,
                int pool, const T* __restrict__ pool_cache, const int* __restrict__ pool_indptr,
                const int* __restrict__ pool_indices, long long pool_pages) {
  bspec::pdl_prologue(7);
  constexpr int W = Shape<ND>::W, D = 32 * ND;
  extern __shared__ __align__(16) float smem_f[];
  const int e = blockIdx.y, kvh = blockIdx.z, G = Hq / Hkv, warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_begin = qo_indptr[e], rows = (qo_indptr[e + 1] - q_begin) * G;
  const int row = (int)(gridDim.x - 1 - blockIdx.x) * warps + warp;
  if (row >= rows) return;
  const int t = q_begin + row / G, h = kvh * G + row % G;
  float* qs = smem_f + warp * (D + W * (D + 2));
  float* part = qs + D;                                     // [W][D]
  float* ml = part + W * D;                                 // [W][2]
  const T* qp = q + (size_t)t * q_row_stride + (size_t)h * hd;
  for (int d = lane; d < hd; d += 32) qs[d] = to_f32(qp[d]);
  const int pos = positions[t], *table = kv_indices + kv_indptr[e];
  int lo = window > 0 ? max(0, pos - window + 1) : 0;
  if (chunk > 0) lo = max(lo, (pos / chunk) * chunk);
  const int before = pool != 0 ? bspec::pooled_seen(pos, window, pool) : 0;
  const size_t k_elems = (size_t)Hkv * page_size * hd;
  const size_t page_elems = k_elems + (v_is_k ? (size_t)0 : (size_t)Hkv * page_size * vd);
  const float slope = slopes != nullptr ? slopes[h] : 0.f;
  float acc[ND], m, l;                                      // l: this lane's keys only
  __syncwarp();
  auto visit = [&](int share, int lo_, int hi_, const int* tab, const T* base, long long pages, bool biased) {
    if (hi_ < lo_) return;
    const bool vec = ((hd | (int)page_elems) & 3) == 0 && ((uintptr_t)base & (4 * sizeof(T) - 1)) == 0;     // keys start on whole quads
    for (int c = lo_ / 32 + (share + W - lo_ / 32 % W) % W; c <= hi_ / 32; c += W) {
      const int key = 32 * c + lane;
      bool on = key >= lo_ && key <= hi_;
      if (on && !bspec::in_range(tab[key / page_size], pages, 107)) on = false;
      long long vo = -1;
      float x = -INFINITY;
      if (on) {
        const size_t page = (size_t)tab[key / page_size] * page_elems;
        const size_t at = (size_t)kvh * page_size + (size_t)(key % page_size);
        const T* kp = base + page + at * hd;
        vo = (long long)(page + (v_is_k ? at * hd : k_elems + at * vd));
        float dot = 0.f;
        if (vec) {
#pragma unroll 4
          for (int d = 0; d < hd; d += 4) {
            const float4 k4 = load4(kp + d), q4 = *reinterpret_cast<const float4*>(qs + d);
            dot = fmaf(q4.x, k4.x, dot);
            dot = fmaf(q4.y, k4.y, dot);
            dot = fmaf(q4.z, k4.z, dot);
            dot = fmaf(q4.w, k4.w, dot);
          }
        } else {
          for (int d = 0; d < hd; ++d) dot = fmaf(qs[d], to_f32(kp[d]), dot);
        }
        x = dot * scale;
        if (softcap > 0.f) x = softcap * tanhf(x / softcap);
        if (biased) x = __fmaf_rn(-slope, (float)(pos - key), x);
      }
      const float top = fmaxf(m, warp_max(x));
      const float p = x == -INFINITY ? 0.f : expf(x - top);
      const float corr = m == top ? 1.f : expf(m - top);
      l = fmaf(l, corr, p);
      if (corr != 1.f) {
#pragma unroll
        for (int i = 0; i < ND; ++i) acc[i] *= corr;
      }
      m = top;
      const int last = min(31, hi_ - 32 * c);
#pragma unroll 4
      for (int k = 0; k <= last; ++k) {
        const float pk = __shfl_sync(0xffffffffu, p, k);
        const long long at = __shfl_sync(0xffffffffu, vo, k);
        if (pk != 0.f) {                                    // an unseen key's value may be anything
#pragma unroll
          for (int i = 0; i < ND; ++i)
            if (lane + 32 * i < vd) acc[i] = fmaf(pk, to_f32(base[at + lane + 32 * i]), acc[i]);
        }
      }
    }
  };
  const int last_share = min(W - 1, max(pos, before - 1) / 32);             // the shares behind it have no chunk
  for (int share = 0; share <= last_share; ++share) {
    m = -INFINITY, l = 0.f;
#pragma unroll
    for (int i = 0; i < ND; ++i) acc[i] = 0.f;
    if (pool < 0) visit(share, 0, before - 1, table, cache, n_pages, slopes != nullptr);
    if (pool > 0) visit(share, 0, before - 1, pool_indices + pool_indptr[e], pool_cache, pool_pages, false);
    visit(share, lo, pos, table, cache, n_pages, slopes != nullptr);
    const float sum = warp_sum(l);
    if (lane == 0) ml[2 * share] = m, ml[2 * share + 1] = sum;
#pragma unroll
    for (int i = 0; i < ND; ++i) part[share * D + lane + 32 * i] = acc[i];
  }
  __syncwarp();
  join_row<T, ND>(part, D, ml, 2, last_share + 1, sink != nullptr ? sink + h : nullptr, out + (size_t)t * out_stride + (size_t)h * vd, vd,
                  gate != nullptr ? gate + (size_t)t * gate_stride + (size_t)h * (gate_per_head ? 1 : vd) : nullptr, gate_per_head, out_scale);
}

template <typename T, int ND, int R, typename... Args>
int launch_shape(int n_entries, int max_rows, int Hkv, cudaStream_t stream, Args... args) {
  static bool set[bspec::kMaxDevices] = {};
  bool& done = set[bspec::current_device()];
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(attn_generic_kernel<T, ND, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_smem(ND, R));
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const dim3 grid((max_rows + R - 1) / R, n_entries, Hkv);
  if (grid.y > 65535 || grid.z > 65535) return (int)cudaErrorInvalidConfiguration;
  BSPEC_LAUNCH((attn_generic_kernel<T, ND, R>), grid, Shape<ND>::W * 32, attn_smem(ND, R), stream, args...);
  return BSPEC_LAUNCH_CHECK();
}

template <typename T, int ND, int R, typename... Args>
int launch_tiles(int n_entries, int max_rows, int Hkv, cudaStream_t stream, Args... args) {
  static bool set[bspec::kMaxDevices] = {};
  bool& done = set[bspec::current_device()];
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(attn_tile_kernel<T, ND, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_tile_smem(ND, R));
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const dim3 grid((max_rows + R - 1) / R, n_entries, Hkv);
  if (grid.y > 65535 || grid.z > 65535) return (int)cudaErrorInvalidConfiguration;
  BSPEC_LAUNCH((attn_tile_kernel<T, ND, R>), grid, Shape<ND>::W * 32, attn_tile_smem(ND, R), stream, args...);
  return BSPEC_LAUNCH_CHECK();
}

template <typename T, int ND, typename... Args>
int launch_rows(int n_entries, int max_rows, int Hkv, cudaStream_t stream, Args... args) {
  const int warps = min(ROW_WARPS, max_rows);
  const dim3 grid((max_rows + warps - 1) / warps, n_entries, Hkv);
  if (grid.y > 65535 || grid.z > 65535) return (int)cudaErrorInvalidConfiguration;
  BSPEC_LAUNCH((attn_row_kernel<T, ND>), grid, warps * 32, attn_row_smem(ND, warps), stream, args...);
  return BSPEC_LAUNCH_CHECK();
}

// R by the rows of the longest portion: 4 for decode steps of groups of up to four heads (a row that is not there costs as
// much as one that is), else 16 (8 where heads of more than 128 numbers would not leave the registers for it).
constexpr int rows_of_block(int width, int max_rows) { return max_rows <= 4 ? 4 : (width <= 128 ? 16 : 8); }

// Whether a row's keys are so few, or the rows so many, that a warp per row is faster.  ``keys``: no request has more (0: not
// known, or a captured step's bound).  us, blocks of R rows / a warp per row; heads are query heads / kv heads x size, float32
// unless said:
//   prompts of up to 32 keys: 7 tokens 32/8 x 64 16 / 6, 24/8 x 128 22 / 8; 64 requests of 20 tokens 260 / 65 and 279 / 73;
//   prompts of up to 64 keys that fill the device: 200 of 60 tokens 2,873 / 1,394 (one of 61 tokens 17 / 26: not);
//   decode up to 64 keys where the device is filled twice: 300 requests of 50 keys 24/8 x 128 372 / 113, 12/2 x 64 69 / 31, 16/1 x 256
//   131 / 113; 64 of 30 keys 24/8 x 128 54 / 26 (32/8 x 64, filled 1.7 times, 18 / 19: not);
//   decode up to 32 keys: groups of more than four heads, R = 16 for them, 64 requests of 30 keys 5/1 x 64 16 / 12, 64/4 x 128
//   47 / 32 (16/1 x 256, R = 8, 29 / 36: not); rows with keys of their own, 32/32 x 96 176 / 23; bfloat16, whose keys a block
//   stages through registers, 32/8 x 64 24 / 20, 16/1 x 256 38 / 35 (4/1 x 16 9.4 / 10.1: not);
//   decode at any length where the device is filled often and most rows of a block are not there: one row of four, 64 requests of
//   1,000 keys 32/32 x 96 1,162 / 736, bfloat16 1,716 / 647 (8/8 x 128, filled 3.5 times, 341 / 746: not); two of four in bfloat16.
bool by_rows(bool bf16, int width, int n_entries, int max_rows, int max_q_len, int Hkv, int keys) {
  const int R = rows_of_block(width, max_rows), nd = width <= 64 ? 2 : (width <= 128 ? 4 : 8), G = max_rows / max_q_len;
  const double full = bspec::sm_count() * (double)((227 * 1024) / (attn_smem(nd, R) + 1024));
  const double waves = (double)((max_rows + R - 1) / R) * n_entries * Hkv / full;
  const bool few = keys > 0 && keys <= 32, some = keys > 0 && keys <= 64;
  if (max_q_len > 1) return few || (some && waves >= (width > 64 ? 2 : 1.5));
  if (few && ((G > 4 && width <= 128) || (G == 1 && (width > 64 || waves >= 1)) || (bf16 && width >= 32))) return true;
  return (some && waves >= 2) || (G == 1 && waves >= (width > 64 ? 5 : 8)) || (G == 2 && bf16 && width > 64 && waves >= 8);
}

template <typename T, typename... Args>
int launch_sizes(int width, int n_entries, int max_rows, int max_q_len, int Hkv, int max_kv_len, cudaStream_t stream, Args... args) {
  if (by_rows(sizeof(T) == 2, width, n_entries, max_rows, max_q_len, Hkv, max_kv_len)) {
    if (width <= 64) return launch_rows<T, 2>(n_entries, max_rows, Hkv, stream, args...);
    if (width <= 128) return launch_rows<T, 4>(n_entries, max_rows, Hkv, stream, args...);
    return launch_rows<T, 8>(n_entries, max_rows, Hkv, stream, args...);
  }
  const int R = rows_of_block(width, max_rows);
  if (R == 4) {
    if (width <= 64) return launch_shape<T, 2, 4>(n_entries, max_rows, Hkv, stream, args...);
    if (width <= 128) return launch_shape<T, 4, 4>(n_entries, max_rows, Hkv, stream, args...);
    return launch_shape<T, 8, 4>(n_entries, max_rows, Hkv, stream, args...);
  }
  if (max_q_len > 1) {
    if (width <= 64) return launch_tiles<T, 2, 16>(n_entries, max_rows, Hkv, stream, args...);
    if (width <= 128) return launch_tiles<T, 4, 16>(n_entries, max_rows, Hkv, stream, args...);
    if constexpr (sizeof(T) == 4) return launch_tiles<T, 8, 8>(n_entries, max_rows, Hkv, stream, args...);
  }
  if (width <= 64) return launch_shape<T, 2, 16>(n_entries, max_rows, Hkv, stream, args...);
  if (width <= 128) return launch_shape<T, 4, 16>(n_entries, max_rows, Hkv, stream, args...);
  return launch_shape<T, 8, 8>(n_entries, max_rows, Hkv, stream, args...);
}
}  // namespace

// q: rows of row stride q_row_stride (elements), heads packed [Hq][hd] at the row start.
// out: [n, Hq*vd].  max_q_len: the longest request portion in the step (sizes the grid).
static int launch_attention_generic(const void* q, long long q_row_stride, void* out, const void* cache, int dtype,
                                    const int* qo_indptr, const int* positions, const int* kv_indptr,
                                    const int* kv_indices, int n_entries, int max_q_len, int Hq, int Hkv, int hd,
                                    int page_size, float scale, int window, long long n_pages, int vd, int chunk,
                                    const float* sink, float softcap, int v_is_k, const float* gate,
                                    long long gate_stride, long long out_stride, float out_scale, int gate_per_head,
                                    const float* slopes, int pool, const void* pool_cache, const int* pool_indptr,
                                    const int* pool_indices, long long pool_pages, int max_kv_len, cudaStream_t stream) {
  if (n_entries <= 0 || max_q_len <= 0) return 0;
  if ((pool != 0 && window <= 0) || (pool > 0 && (v_is_k || pool_cache == nullptr || pool_indptr == nullptr)))
    return (int)cudaErrorInvalidValue;
  if (v_is_k && vd != hd) return (int)cudaErrorInvalidValue;
  if (hd > MAX_HD || hd <= 0 || vd > MAX_HD || vd <= 0 || Hq % Hkv != 0) return (int)cudaErrorInvalidValue;
  const long long max_rows = (long long)max_q_len * (Hq / Hkv);
  if (max_rows > (1 << 30)) return (int)cudaErrorInvalidConfiguration;
  const int width = hd > vd ? hd : vd;
  if (dtype == BSPEC_F32)
    return launch_sizes<float>(width, n_entries, (int)max_rows, max_q_len, Hkv, max_kv_len, stream, (const float*)q, q_row_stride, (float*)out,
                               (const float*)cache, qo_indptr, positions, kv_indptr, kv_indices, Hq, Hkv, hd, page_size, scale,
                               window, n_pages, vd, chunk, sink, softcap, v_is_k, gate, gate_stride, out_stride, out_scale,
                               gate_per_head, slopes, pool, (const float*)pool_cache, pool_indptr, pool_indices, pool_pages);
  return launch_sizes<__nv_bfloat16>(width, n_entries, (int)max_rows, max_q_len, Hkv, max_kv_len, stream, (const __nv_bfloat16*)q, q_row_stride,
                                     (__nv_bfloat16*)out, (const __nv_bfloat16*)cache, qo_indptr, positions, kv_indptr, kv_indices,
                                     Hq, Hkv, hd, page_size, scale, window, n_pages, vd, chunk, sink, softcap, v_is_k, gate,
                                     gate_stride, out_stride, out_scale, gate_per_head, slopes, pool, (const __nv_bfloat16*)pool_cache,
                                     pool_indptr, pool_indices, pool_pages);
}

BSPEC_API int bspec_attention_generic(const void* q, long long q_row_stride, void* out, const void* cache, int dtype,
                                      const int* qo_indptr, const int* positions, const int* kv_indptr,
                                      const int* kv_indices, int n_entries, int max_q_len, int Hq, int Hkv, int hd,
                                      int page_size, float scale, int window, long long n_pages,
                                      cudaStream_t stream) {
  return launch_attention_generic(q, q_row_stride, out, cache, dtype, qo_indptr, positions, kv_indptr, kv_indices,
                                  n_entries, max_q_len, Hq, Hkv, hd, page_size, scale, window, n_pages, hd, 0, nullptr,
                                  0.f, 0, nullptr, 0, (long long)Hq * hd, 1.f, 0, nullptr, 0, nullptr, nullptr, nullptr,
                                  0, 0, stream);
}

// The same with values of their own size ``vd``, a chunk mask (0: none), a sink per query head (null: none), a soft
// cap on the scores (0: none), values that are the keys, a sigmoid gate on the output (per number, or per head), an
// output scale and stride, a distance bias (slopes per query head, null: none) and pooled blocks or kept first tokens
// before the window (pool > 0 or < 0; 0: none).  ``max_kv_len``: no request has more keys (0: not known).
BSPEC_API int bspec_attention_masked(const void* q, long long q_row_stride, void* out, const void* cache, int dtype,
                                     const int* qo_indptr, const int* positions, const int* kv_indptr,
                                     const int* kv_indices, int n_entries, int max_q_len, int Hq, int Hkv, int hd,
                                     int vd, int page_size, float scale, int window, int chunk, const float* sink,
                                     long long n_pages, float softcap, int v_is_k, const float* gate,
                                     long long gate_stride, long long out_stride, float out_scale,
                                     int gate_per_head, const float* slopes, int pool, const void* pool_cache,
                                     const int* pool_indptr, const int* pool_indices, long long pool_pages,
                                     int max_kv_len, cudaStream_t stream) {
  return launch_attention_generic(q, q_row_stride, out, cache, dtype, qo_indptr, positions, kv_indptr, kv_indices,
                                  n_entries, max_q_len, Hq, Hkv, hd, page_size, scale, window, n_pages, vd, chunk, sink,
                                  softcap, v_is_k, gate, gate_stride, out_stride, out_scale, gate_per_head, slopes, pool,
                                  pool_cache, pool_indptr, pool_indices, pool_pages, max_kv_len, stream);
}

// ---------------------------------------------------------------- q/k/v preparation
// From the float32 rows of the fused projection [q: Hq*hd | k: Hkv*hd | v: Hkv*vd]: add the bias (if any), rotate the
// first ``rot`` numbers of every q and k head (pair (i, i + rot/2), or (2i, 2i+1) with ``interleaved``; cosine and
// sine times ``magnitude``), divide every q and k head by its root mean square (``norm_eps`` > 0; none otherwise; times ``q_norm_w`` / ``k_norm_w``,
// a weight per number of a head, when given; before the rotation with ``norm_first``),
// all in float32; then write q to ``q_out`` [n, Hq*hd] and k and v into the cache page of the token's position.
// Rows of the input have stride ``ld`` (they may hold more columns).  vd == 0: there are no values (they are the
// keys); a page then holds keys only.  One warp per head.  ``pool`` P > 0 (only for steps whose entries have one token
// each): a token that completes a block of P also leaves the block's mean key and value, of the rows as the cache
// holds them, in the pooled pages; larger portions take ``pool_append`` below after this kernel.
namespace {
constexpr int PREP_WARPS = 8;

// Mean over the ``pool`` rows (from position p0, pages through ``table``) of one column of a kv head, in row order:
// float32 sum, one division, the cache's rounding.  ``part``: the column's offset in a page's row 0, ``width`` the
// distance from row to row.
template <typename T>
__device__ __forceinline__ float pooled_mean(const T* __restrict__ cache, const int* __restrict__ table, size_t page_elems,
                                             size_t part, int width, int p0, int pool, int page_size,
                                             long long n_pages) {
  float s = 0.f;
#pragma unroll 8
  for (int r = 0; r < pool; ++r) {
    const int p = p0 + r, page = table[p / page_size];
    if (bspec::in_range(page, n_pages, 116))
      s += to_f32(cache[(size_t)page * page_elems + part + (size_t)(p % page_size) * width]);
  }
  return s / (float)pool;
}

__device__ __forceinline__ void row4(const float* p, float (&f)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
}
__device__ __forceinline__ void row4(const __nv_bfloat16* p, float (&f)[4]) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&v.x), b = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
  f[0] = __low2float(a), f[1] = __high2float(a), f[2] = __low2float(b), f[3] = __high2float(b);
}

// The same for four columns at once (head sizes that are multiples of 4); each column's arithmetic is the same.
template <typename T>
__device__ __forceinline__ void pooled_mean4(float (&m)[4], const T* __restrict__ cache, const int* __restrict__ table,
                                             size_t page_elems, size_t part, int width, int p0, int pool, int page_size,
                                             long long n_pages) {
  m[0] = m[1] = m[2] = m[3] = 0.f;
#pragma unroll 8
  for (int r = 0; r < pool; ++r) {
    const int p = p0 + r, page = table[p / page_size];
    if (bspec::in_range(page, n_pages, 116)) {
      float v[4];
      row4(cache + (size_t)page * page_elems + part + (size_t)(p % page_size) * width, v);
#pragma unroll
      for (int c = 0; c < 4; ++c) m[c] += v[c];
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) m[c] = m[c] / (float)pool;
}

__device__ __forceinline__ void prep_sincos(int pos, const float* __restrict__ inv_freq, int half, int j, float* s,
                                            float* c) {
  const double f = (double)inv_freq[j] + (double)inv_freq[half + j];
  double a = (double)pos * f;
  a -= 6.283185307179586476925286766559 * rint(a * 0.15915494309189533576888376337251);
  sincosf((float)a, s, c);
}

__device__ __forceinline__ void prep_store4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void prep_store4(__nv_bfloat16* p, float a, float b, float c, float d) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  uint2 v;
  v.x = *reinterpret_cast<const uint32_t*>(&lo);
  v.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = v;
}

template <typename T>
__global__ void __launch_bounds__(PREP_WARPS * 32)
qkv_prepare_kernel(const float* __restrict__ qkv, long long ld, int Hq, int Hkv, int hd, int vd, const void* __restrict__ bias,
                   int bias_dtype, const float* __restrict__ inv_freq, int rot, int interleaved, float magnitude,
                   float norm_eps, const int* __restrict__ positions, const int* __restrict__ tok_entry,
                   const int* __restrict__ kv_indptr, const int* __restrict__ kv_indices, T* __restrict__ q_out,
                   T* __restrict__ cache, int page_size, int write_kv, long long n_pages,
                   const void* __restrict__ q_norm_w, const void* __restrict__ k_norm_w, int norm_w_dtype,
                   int norm_first, int pool, T* __restrict__ pool_cache, const int* __restrict__ pool_indptr,
                   const int* __restrict__ pool_indices, long long pool_pages) {
  bspec::pdl_prologue(19);
  __shared__ __align__(16) float xs[PREP_WARPS][MAX_HD];
  __shared__ float cs[MAX_HD];                                // [rot/2] cosines, then [rot/2] sines, of this token
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slot = blockIdx.y * PREP_WARPS + warp;            // q heads, then k heads, then v heads
  const int pos = positions[t];
  const bool has = slot < Hq + Hkv + (vd > 0 ? Hkv : 0);
  const bool is_v = slot >= Hq + Hkv;
  const int width = is_v ? vd : hd;
  const int col0 = is_v ? (Hq + Hkv) * hd + (slot - Hq - Hkv) * vd : slot * hd;
  const float* src = qkv + (size_t)t * ld + (has ? col0 : 0);
  float* x = xs[warp];
  const bool vec = ((hd | vd | (int)ld) & 3) == 0;           // every head starts on a 16-byte boundary: four numbers per lane
  // the head's numbers are asked for first, so that their way from memory runs under the angles' arithmetic
  float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
  if (has && vec) {
    if (4 * lane < width) v0 = *reinterpret_cast<const float4*>(src + 4 * lane);
    if (4 * lane + 128 < width) v1 = *reinterpret_cast<const float4*>(src + 4 * lane + 128);
  }
  if (blockIdx.y * PREP_WARPS < Hq + Hkv) {                   // the block holds a q or k head: the angles once for all
    const int half = rot / 2;
    for (int j = threadIdx.x; j < half; j += blockDim.x) {
      float sn, c;
      prep_sincos(pos, inv_freq, half, j, &sn, &c);
      cs[j] = c * magnitude;
      cs[half + j] = sn * magnitude;
    }
  }
  __syncthreads();
  if (!has) return;
  if (vec) {
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const int d = 4 * lane + 128 * part;
      if (d < width) {
        float4 v = part ? v1 : v0;
        if (bias != nullptr) {
          v.x += load_as_f32(bias, bias_dtype, (size_t)col0 + d);
          v.y += load_as_f32(bias, bias_dtype, (size_t)col0 + d + 1);
          v.z += load_as_f32(bias, bias_dtype, (size_t)col0 + d + 2);
          v.w += load_as_f32(bias, bias_dtype, (size_t)col0 + d + 3);
        }
        *reinterpret_cast<float4*>(x + d) = v;
      }
    }
  } else {
    for (int d = lane; d < width; d += 32)
      x[d] = src[d] + (bias != nullptr ? load_as_f32(bias, bias_dtype, (size_t)col0 + d) : 0.f);
  }
  __syncwarp();
  if (!is_v) {
    // every q and k head divided by its root mean square, times a weight per number when one is given (the same
    // for all heads); before the rotation (norm_first) or after it
    const void* nw = slot < Hq ? q_norm_w : k_norm_w;
    auto normalise = [&]() {
      float ss = 0.f;
      for (int d = lane; d < hd; d += 32) ss += x[d] * x[d];
      ss = warp_sum(ss);
      const float r = 1.f / sqrtf(ss / (float)hd + norm_eps);
      for (int d = lane; d < hd; d += 32) x[d] = x[d] * r * (nw != nullptr ? load_as_f32(nw, norm_w_dtype, d) : 1.f);
      __syncwarp();
    };
    if (norm_eps > 0.f && norm_first) normalise();
    const int half = rot / 2;
    for (int j = lane; j < half; j += 32) {
      const float c = cs[j], sn = cs[half + j];
      const int a = interleaved ? 2 * j : j, b = interleaved ? 2 * j + 1 : j + half;
      const float u = x[a], v = x[b];
      x[a] = u * c - v * sn;
      x[b] = v * c + u * sn;
    }
    __syncwarp();
    if (norm_eps > 0.f && !norm_first) normalise();
  }
  const float r = 1.f;
  T* dst = nullptr;
  if (slot < Hq) {
    dst = q_out + ((size_t)t * Hq + slot) * hd;
  } else if (write_kv) {
    const int e = tok_entry[t];
    if (bspec::in_range(pos / page_size, kv_indptr[e + 1] - kv_indptr[e], 113)) {
      const int page = kv_indices[kv_indptr[e] + pos / page_size];
      if (bspec::in_range(page, n_pages, 114)) {
        const size_t k_elems = (size_t)Hkv * page_size * hd;
        const size_t page_elems = k_elems + (size_t)Hkv * page_size * vd;
        const int row = pos % page_size;
        dst = cache + (size_t)page * page_elems +
              (is_v ? k_elems + ((size_t)(slot - Hq - Hkv) * page_size + row) * vd
                    : ((size_t)(slot - Hq) * page_size + row) * hd);
      }
    }
  }
  if (dst != nullptr) {
    if (vec) {
      for (int d = 4 * lane; d < width; d += 128) {
        const float4 v = *reinterpret_cast<const float4*>(x + d);
        prep_store4(dst + d, v.x * r, v.y * r, v.z * r, v.w * r);
      }
    } else {
      for (int d = lane; d < width; d += 32) dst[d] = from_f32<T>(x[d] * r);
    }
  }
  if (pool > 0 && dst != nullptr && slot >= Hq && (pos + 1) % pool == 0) {
    // this token completes its block, and the block's other rows are of earlier steps
    __syncwarp();                                            // the row just written is read back by other lanes
    const int e = tok_entry[t], b = pos / pool;
    const int* ptab = pool_indices + pool_indptr[e];
    const size_t k_elems = (size_t)Hkv * page_size * hd, page_elems = k_elems + (size_t)Hkv * page_size * vd;
    const size_t head = is_v ? k_elems + (size_t)(slot - Hq - Hkv) * page_size * vd : (size_t)(slot - Hq) * page_size * hd;
    if (bspec::in_range(b / page_size, pool_indptr[e + 1] - pool_indptr[e], 117) &&
        bspec::in_range(ptab[b / page_size], pool_pages, 118)) {
      T* to = pool_cache + (size_t)ptab[b / page_size] * page_elems + head + (size_t)(b % page_size) * width;
      if (vec) {
        for (int d = 4 * lane; d < width; d += 128) {
          float m[4];
          pooled_mean4<T>(m, cache, kv_indices + kv_indptr[e], page_elems, head + d, width, b * pool, pool, page_size, n_pages);
          prep_store4(to + d, m[0], m[1], m[2], m[3]);
        }
        return;
      }
      for (int d = lane; d < width; d += 32)
        to[d] = from_f32<T>(pooled_mean<T>(cache, kv_indices + kv_indptr[e], page_elems, head + d, width, b * pool, pool,
                                           page_size, n_pages));
    }
  }
}

// The pooled entries of the blocks that a step's portions complete: block (x, e, z) takes the x-th such block of
// entry e; a thread per column (VEC: per four columns) of [k of every kv head | v of every kv head].
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
pool_append_kernel(const T* __restrict__ cache, const int* __restrict__ qo_indptr, const int* __restrict__ positions,
                   const int* __restrict__ kv_indptr, const int* __restrict__ kv_indices, T* __restrict__ pool_cache,
                   const int* __restrict__ pool_indptr, const int* __restrict__ pool_indices, int Hkv, int hd, int vd,
                   int page_size, int pool, long long n_pages, long long pool_pages) {
  bspec::pdl_prologue(21);
  const int e = blockIdx.y;
  const int t0 = qo_indptr[e], nt = qo_indptr[e + 1] - t0;
  if (nt <= 0) return;
  const int pos0 = positions[t0];
  const int b = pos0 / pool + (int)blockIdx.x;
  if ((long long)(b + 1) * pool > pos0 + nt) return;
  const int col = (VEC ? 4 : 1) * (blockIdx.z * blockDim.x + threadIdx.x);
  if (col >= Hkv * (hd + vd)) return;
  const bool is_v = col >= Hkv * hd;
  const int width = is_v ? vd : hd, c = is_v ? col - Hkv * hd : col;
  const int g = c / width, d = c - g * width;
  const size_t k_elems = (size_t)Hkv * page_size * hd, page_elems = k_elems + (size_t)Hkv * page_size * vd;
  const size_t head = (is_v ? k_elems : (size_t)0) + (size_t)g * page_size * width;
  const int* ptab = pool_indices + pool_indptr[e];
  if (!bspec::in_range(b / page_size, pool_indptr[e + 1] - pool_indptr[e], 117) ||
      !bspec::in_range(ptab[b / page_size], pool_pages, 118))
    return;
  T* to = pool_cache + (size_t)ptab[b / page_size] * page_elems + head + (size_t)(b % page_size) * width + d;
  if (VEC) {
    float m[4];
    pooled_mean4<T>(m, cache, kv_indices + kv_indptr[e], page_elems, head + d, width, b * pool, pool, page_size, n_pages);
    prep_store4(to, m[0], m[1], m[2], m[3]);
  } else {
    *to = from_f32<T>(pooled_mean<T>(cache, kv_indices + kv_indptr[e], page_elems, head + d, width, b * pool, pool,
                                     page_size, n_pages));
  }
}
}  // namespace

// Portions of any length; max_q_len: the longest of the step.
BSPEC_API int bspec_pool_append(const void* cache, int dtype, const int* qo_indptr, const int* positions,
                                const int* kv_indptr, const int* kv_indices, void* pool_cache, const int* pool_indptr,
                                const int* pool_indices, int n_entries, int max_q_len, int Hkv, int hd, int vd,
                                int page_size, int pool, long long n_pages, long long pool_pages, cudaStream_t stream) {
  if (n_entries <= 0 || max_q_len <= 0) return 0;
  if (pool <= 0 || Hkv <= 0 || hd <= 0 || vd < 0 || page_size <= 0 || n_entries > 65535) return (int)cudaErrorInvalidValue;
  const bool vec = hd % 4 == 0 && vd % 4 == 0;
  const int items = Hkv * (hd + vd) / (vec ? 4 : 1), threads = items >= 256 ? 256 : ((items + 31) / 32) * 32;
  const dim3 grid((max_q_len + pool - 1) / pool, n_entries, (items + threads - 1) / threads);
  if (grid.z > 65535) return (int)cudaErrorInvalidConfiguration;
#define LP(T, V)                                                                                                     \
  BSPEC_LAUNCH((pool_append_kernel<T, V>), grid, threads, 0, stream, (const T*)cache, qo_indptr, positions, kv_indptr, \
               kv_indices, (T*)pool_cache, pool_indptr, pool_indices, Hkv, hd, vd, page_size, pool, n_pages, pool_pages)
  if (dtype == BSPEC_F32) { if (vec) LP(float, true); else LP(float, false); }
  else { if (vec) LP(__nv_bfloat16, true); else LP(__nv_bfloat16, false); }
#undef LP
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_API int bspec_qkv_prepare(const float* qkv, long long ld, int n, int Hq, int Hkv, int hd, int vd, const void* bias,
                                int bias_dtype, const float* inv_freq, int rot, int interleaved, float magnitude,
                                float norm_eps, const int* positions, const int* tok_entry, const int* kv_indptr,
                                const int* kv_indices, void* q_out, void* cache, int dtype, int page_size, int write_kv,
                                long long n_pages, const void* q_norm_w, const void* k_norm_w, int norm_w_dtype,
                                int norm_first, int pool, void* pool_cache, const int* pool_indptr,
                                const int* pool_indices, long long pool_pages, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (pool < 0 || (pool > 0 && (pool_cache == nullptr || pool_indptr == nullptr || !write_kv)))
    return (int)cudaErrorInvalidValue;
  if (hd <= 0 || hd > MAX_HD || vd < 0 || vd > MAX_HD || ld < (long long)(Hq + Hkv) * hd + (long long)Hkv * vd || rot < 0 || rot > hd || rot % 2 != 0 ||
      (rot > 0 && inv_freq == nullptr))
    return (int)cudaErrorInvalidValue;
  const dim3 grid(n, (Hq + 2 * Hkv + PREP_WARPS - 1) / PREP_WARPS);
  if (grid.y > 65535) return (int)cudaErrorInvalidConfiguration;
  if (dtype == BSPEC_F32)
    BSPEC_LAUNCH((qkv_prepare_kernel<float>), grid, PREP_WARPS * 32, 0, stream, qkv, ld, Hq, Hkv, hd, vd, bias, bias_dtype,
                 inv_freq, rot, interleaved, magnitude, norm_eps, positions, tok_entry, kv_indptr, kv_indices,
                 (float*)q_out, (float*)cache, page_size, write_kv, n_pages, q_norm_w, k_norm_w, norm_w_dtype, norm_first,
                 pool, (float*)pool_cache, pool_indptr, pool_indices, pool_pages);
  else
    BSPEC_LAUNCH((qkv_prepare_kernel<__nv_bfloat16>), grid, PREP_WARPS * 32, 0, stream, qkv, ld, Hq, Hkv, hd, vd, bias,
                 bias_dtype, inv_freq, rot, interleaved, magnitude, norm_eps, positions, tok_entry, kv_indptr,
                 kv_indices, (__nv_bfloat16*)q_out, (__nv_bfloat16*)cache, page_size, write_kv, n_pages, q_norm_w, k_norm_w,
                 norm_w_dtype, norm_first, pool, (__nv_bfloat16*)pool_cache, pool_indptr, pool_indices, pool_pages);
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_DEFINE_TRACE_SETTER(bspec_trace_set_attention_generic)
BSPEC_DEFINE_BOUNDS_REPORT(bspec_bounds_report_attention_generic)
