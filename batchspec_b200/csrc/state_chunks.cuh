// Recurrences with one matrix of state per head, S [key rows x value columns] float32, taken in chunks of 64 tokens: whatever a
// chunk contributes that does not depend on S is a product of matrices of 64 tokens and up to 128 numbers, formed by all SMs at
// once, and only what is left goes from chunk to chunk (the chunkwise form of linear attention with decay, as in RetNet, Sun et al.
// 2023).  Float32 in packed multiply-adds.  Lightning attention (state_mixers.cu)
// takes it; the delta rule does not: its chunks also need a triangular inverse and the products with it, 115 + 176 + 101 us a
// layer at 3 prompts of 4,000 tokens in all against 399 + 35 us by tiles of eight tokens, and the pass was no faster.
#pragma once
#include "state_tiles.cuh"

namespace bspec {

constexpr int CH = 64, CH_W = 128, CH_LD = CH_W + 4, CH_AT = CH + 4, CH_SL = 32, CH_THREADS = 256;     // tokens; numbers of a head at most
constexpr int CH_FROM = 512;                         // no chunks in steps whose longest portion is shorter

// Where chunk i of entry e has its scratch (times heads): chunks of different entries never meet.
__host__ __device__ __forceinline__ size_t chunk_slot(int q_begin, int e, int i) { return (size_t)(q_begin / CH + e + i); }
inline long long chunk_slots(int n, int n_entries) { return n / CH + n_entries + 1; }
// The entry whose slots hold ``slot``: the last one that begins at or before it.
__device__ __forceinline__ int chunk_entry(const int* __restrict__ qo_indptr, int n_entries, int slot) {
  int lo = 0, hi = n_entries;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((int)chunk_slot(qo_indptr[mid], mid, 0) <= slot) lo = mid; else hi = mid;
  }
  return lo;
}
// Heads that fill most of the 128 x 128 numbers which the products are laid out for.
inline bool chunk_sizes(int dim, int vdim) { return dim <= CH_W && vdim <= CH_W && dim % 4 == 0 && dim * vdim >= 96 * 96; }

// acc[a][b] = (even, odd) parts of S^T q for tokens tb + a (a < 8: a warp's) and columns lane + 32 b.  qs [CH][CH_LD] queries, S
// [vdim][dim] in memory, ss [CH_W][CH_SL + 4] shared memory for a slice of 32 key rows.  All threads of the block.
__device__ __forceinline__ void chunk_read_state(unsigned long long (&acc)[8][4], const float* qs, float* ss, const float* __restrict__ S,
                                                 int dim, int vdim, int tb, int lane) {
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0ull;
  for (int r0 = 0; r0 < dim; r0 += CH_SL) {
    if (r0 > 0) __syncthreads();
    for (int x = threadIdx.x; x < CH_W * (CH_SL / 4); x += CH_THREADS) {
      const int j = x / (CH_SL / 4), r = x % (CH_SL / 4) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < vdim && r0 + r < dim) v = *reinterpret_cast<const float4*>(S + (size_t)j * dim + r0 + r);
      *reinterpret_cast<float4*>(ss + j * (CH_SL + 4) + r) = v;
    }
    __syncthreads();
#pragma unroll 2
    for (int r = 0; r < CH_SL; r += 4) {
      ulonglong2 sj[4];
#pragma unroll
      for (int b = 0; b < 4; ++b) sj[b] = *reinterpret_cast<const ulonglong2*>(ss + (lane + 32 * b) * (CH_SL + 4) + r);
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(qs + (tb + a) * CH_LD + r0 + r);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          fma_pair(acc[a][b], q.x, sj[b].x);
          fma_pair(acc[a][b], q.y, sj[b].y);
        }
      }
    }
  }
}

// o[p][b] += sum_(s <= t) M[t][s] value(s, b) for the tokens t = tb + 2 p, tb + 2 p + 1, M's columns as rows at[s][t].  What a
// later token holds may be anything: it has no part.
template <typename Value>
__device__ __forceinline__ void chunk_below(unsigned long long (&o)[4][4], const float* at, int tb, Value value) {
  auto rows_of = [&](int s, unsigned long long (&a)[4]) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(at + s * CH_AT + tb), a1 = *reinterpret_cast<const ulonglong2*>(at + s * CH_AT + tb + 4);
    a[0] = a0.x, a[1] = a0.y, a[2] = a1.x, a[3] = a1.y;
  };
#pragma unroll 2
  for (int s = 0; s < tb; ++s) {                     // tokens before this warp's
    unsigned long long a[4];
    rows_of(s, a);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float v = value(s, b);
      const unsigned long long v2 = pair_of(v, v);
#pragma unroll
      for (int p = 0; p < 4; ++p) fma_pair(o[p][b], a[p], v2);
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {                      // its own
    unsigned long long a[4];
    rows_of(tb + k, a);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float v = value(tb + k, b);
#pragma unroll
      for (int p = k / 2; p < 4; ++p) fma_pair(o[p][b], a[p], pair_of(k <= 2 * p ? v : 0.f, v));
    }
  }
}

// o to rows of ``ld`` floats, columns lane + 32 b below ``width``, tokens below ``cnt``
__device__ __forceinline__ void chunk_write(const unsigned long long (&o)[4][4], float* __restrict__ dst, long long ld, int width, int cnt,
                                            int tb, int lane) {
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int t = tb + 2 * p, j = lane + 32 * b;
      float x, y;
      halves_of(o[p][b], x, y);
      if (j < width && t < cnt) dst[t * ld + j] = x;
      if (j < width && t + 1 < cnt) dst[(t + 1) * ld + j] = y;
    }
}
}  // namespace bspec
