// Latent attention of long portions (bfloat16) with keys and values per head: the entries [c | kr] that a portion sees are
// gathered from their pages, one matrix product forms every head's key and value parts [Wuk_h; Wuv_h] c of them, and a
// flash attention on the 5th-generation tensor cores runs over those.  Per (query, key) pair and head that is
// dim + rot_dim + 2 vdim = 448 multiply-adds (the weights enter the product with the values as two bfloat16 numbers, the
// rounded weight and the rounding's remainder) where attention in the latent space takes rank + rot_dim + 2 rank = 1,600,
// and a head's accumulator fits tensor memory twice.  The products per entry cost what the queries' way into the latent
// space and the outputs' way out of it cost per token otherwise, so it pays as soon as a portion has some tens of tokens
// (a step of four layers of 16 heads, latent 512, us, here / in the latent space: 64 tokens 396 / 396, 256 459 / 516, 1,024
// 814 / 1,466; 64 after 2,048 632 / 1,277).  Keys and values per head are rounded to bfloat16 here, the queries' and outputs' latents
// there; both are as far from 64 bits.  Heads of 128 + 64 / 128 numbers only; others stay in the latent space.
//
//   latent_gather_kernel   pages -> rows: cbuf [T, R], krbuf [T, P].  A portion's rows begin at a multiple of 64 and are
//                          filled up to one with zeros, T rows in all; base[e] is the first row of entry e.
//   latent_prompt_kernel   one persistent CTA per SM; items of 256 tokens of one request and one head, as two Q tiles of
//                          128 rows with a softmax warpgroup each, keys in tiles of 64:
//     warp 0      TMA: the Q tiles, and K (dim from the product, rot_dim from the entries) and V tiles in rings of three;
//     warps 1, 10 one thread each issues S = Q K^T for its Q tile, two key tiles ahead, into one of two buffers, and
//                 O += P_hi V + P_lo V with P read from tensor memory;
//     warps 2-9   one thread per row: scale, mask, online softmax in float32; the weights' two parts go over the S they
//                 came from (32 columns each).
//   Tensor memory: 2 x 2 S buffers of 64 columns, 2 O accumulators of 128.  Every wait is bounded.
// Bound by the softmax between the two products.  2,048 tokens of 16 heads: 66 us, 325 TFLOP/s (455 with the weights' second part);
// latent_attn_mma for the same 636 us.
#include "umma.cuh"
#include <math.h>

using namespace bspec;

namespace {

constexpr int DK = 128, PR = 64, DV = 128;           // unrotated and rotated query/key numbers and value numbers per head
constexpr int ROWS = 128, QT = 2, KT = 64, STAGES = 3;
constexpr int MMA_WARP_1 = 2 + 4 * QT, THREADS = 32 * (3 + 4 * QT);
constexpr int SUBQ = ROWS * 64 * 2, SUBK = KT * 64 * 2;               // bytes of 64 columns of a Q and of a key tile
constexpr int Q_BYTES = 3 * SUBQ, K_BYTES = 3 * SUBK, V_BYTES = 2 * SUBK;
constexpr int SMEM = 1024 + QT * Q_BYTES + STAGES * (K_BYTES + V_BYTES) + 256;

// What is asked of entry e: its tokens, the first key its tokens see (down to a multiple of 64), how many rows of keys.
struct Span {
  int q_begin, q_len, pos0, k_first, rows;
};
__device__ __forceinline__ Span span_of(int e, const int* __restrict__ qo_indptr, const int* __restrict__ positions, int window,
                                        int min_q) {
  Span s;
  s.q_begin = qo_indptr[e];
  s.q_len = qo_indptr[e + 1] - s.q_begin;
  s.rows = 0;
  s.pos0 = s.k_first = 0;
  if (s.q_len >= min_q) {
    s.pos0 = positions[s.q_begin];
    s.k_first = bspec::mask_lo(s.pos0, window) / KT * KT;
    s.rows = (s.pos0 + s.q_len - s.k_first + KT - 1) / KT * KT;
  }
  return s;
}

// Block b fills rows 64 b .. 64 b + 63.  Every block finds its entry by adding up the entries' rows, 256 at a time.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const __nv_bfloat16* __restrict__ cache, const int* __restrict__ qo_indptr, const int* __restrict__ positions,
                     const int* __restrict__ kv_indptr, const int* __restrict__ kv_indices, int n_entries, int R, int page_size,
                     int window, int min_q, __nv_bfloat16* __restrict__ cbuf, __nv_bfloat16* __restrict__ krbuf,
                     int* __restrict__ base, long long n_pages) {
  bspec::pdl_prologue(45);
  __shared__ int warp_rows[8], found[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, want = blockIdx.x * KT;
  if (tid == 0) found[0] = -1;
  int before = 0;
  for (int e0 = 0; e0 < n_entries; e0 += 256) {
    const int e = e0 + tid;
    const int rows = e < n_entries ? span_of(e, qo_indptr, positions, window, min_q).rows : 0;
    int sum = rows;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    __syncthreads();
    if (lane == 31) warp_rows[warp] = sum;
    __syncthreads();
    int first = before + sum - rows, all = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) first += warp_rows[w];
      all += warp_rows[w];
    }
    if (rows > 0 && want >= first && want < first + rows) {
      found[0] = e;
      found[1] = first;
    }
    if (blockIdx.x == 0 && e < n_entries) base[e] = first;
    before += all;
  }
  __syncthreads();
  const int e = found[0];
  if (e < 0) return;
  const Span s = span_of(e, qo_indptr, positions, window, min_q);
  const int key0 = s.k_first + want - found[1], k_end = s.pos0 + s.q_len, k_lo = bspec::mask_lo(s.pos0, window);
  const int* table = kv_indices + kv_indptr[e];
  const int D = R + PR, chunks = D / 8;
  for (int i = tid; i < KT * chunks; i += 256) {
    const int r = i / chunks, c = (i - r * chunks) * 8, key = key0 + r;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (key >= k_lo && key < k_end) {                          // (entries before k_lo may have been given back)
      const int page = table[key / page_size];
      if (bspec::in_range(page, n_pages, 112))
        v = *reinterpret_cast<const uint4*>(cache + ((size_t)page * page_size + key % page_size) * D + c);
    }
    __nv_bfloat16* dst = c < R ? cbuf + (size_t)(want + r) * R + c : krbuf + (size_t)(want + r) * PR + (c - R);
    *reinterpret_cast<uint4*>(dst) = v;
  }
}

struct Params {
  __nv_bfloat16* out;              // [.., token, head, DV] with strides
  long long o_row, o_head;
  const int* qo_indptr;
  const int* positions;
  const int* base;
  const float* sink;
  int* status;
  int n_entries, n_items, head0, heads, window, min_q;
  float scale_log2;
};

struct Item {
  Span s;
  int h, row0, base, k_begin, n_kt[QT], n_tiles, k_end_t[QT];
};

// Items in the order they are dealt: head fastest, then request, then blocks of 256 tokens from the last (most keys) to
// the first.  False: the index names no work.
__device__ __forceinline__ bool load_item(Item& it, int idx, const Params& p) {
  const int hl = idx % p.heads, ez = idx / p.heads, e = ez % p.n_entries, z = ez / p.n_entries;
  it.s = span_of(e, p.qo_indptr, p.positions, p.window, p.min_q);
  if (it.s.rows == 0) return false;
  const int blocks = (it.s.q_len + QT * ROWS - 1) / (QT * ROWS);
  if (z >= blocks) return false;
  it.h = hl;
  it.row0 = (blocks - 1 - z) * QT * ROWS;
  it.base = p.base[e];
  it.k_begin = bspec::mask_lo(it.s.pos0 + it.row0, p.window) / KT * KT;
  it.n_tiles = 0;
#pragma unroll
  for (int t = 0; t < QT; ++t) {
    const int r = it.row0 + t * ROWS;
    it.n_kt[t] = 0;
    it.k_end_t[t] = it.k_begin;
    if (r < it.s.q_len) {
      it.k_end_t[t] = it.s.pos0 + min(it.s.q_len, r + ROWS);
      it.n_kt[t] = (it.k_end_t[t] - it.k_begin + KT - 1) / KT;
    }
    it.n_tiles = max(it.n_tiles, it.n_kt[t]);
  }
  return true;
}
// The n-th item of this CTA: rounds of gridDim.x items, every second one dealt backwards, so that the CTA with the longest
// item of a round has the shortest of the next.
__device__ __forceinline__ int item_of(int n) {
  return n * (int)gridDim.x + ((n & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
}

__global__ void __launch_bounds__(THREADS, 1)
latent_prompt_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map,
                     const __grid_constant__ CUtensorMap kr_map, const Params p) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* Qs = smem;
  unsigned char* Ks = Qs + QT * Q_BYTES;
  unsigned char* Vs = Ks + STAGES * K_BYTES;
  uint64_t* k_full = reinterpret_cast<uint64_t*>(Vs + STAGES * V_BYTES);
  uint64_t* k_empty = k_full + STAGES;
  uint64_t* v_full = k_empty + STAGES;
  uint64_t* v_empty = v_full + STAGES;
  uint64_t* s_full = v_empty + STAGES;               // [QT][2]
  uint64_t* p_ready = s_full + 2 * QT;               // [QT][2]
  uint64_t* pv_done = p_ready + 2 * QT;              // [QT][2]
  uint64_t* q_ready = pv_done + 2 * QT;              // [QT]
  uint64_t* q_free = q_ready + QT;                   // [QT]  every S product of the item has read its Q tile
  uint64_t* o_free = q_free + QT;                    // [QT]  the item's O has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_free + QT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* const status = p.status;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(k_empty + s, QT);
      mbar_init(v_full + s, 1);
      mbar_init(v_empty + s, QT);
    }
    for (int i = 0; i < 2 * QT; ++i) {
      mbar_init(s_full + i, 1);
      mbar_init(p_ready + i, 4);
      mbar_init(pv_done + i, 1);
    }
    for (int i = 0; i < QT; ++i) {
      mbar_init(q_ready + i, 1);
      mbar_init(q_free + i, 1);
      mbar_init(o_free + i, 4);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bspec::pdl_wait();
  Item it;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t kn = 0, vn = 0, qn[QT] = {0, 0};
      bool ok = true;
      for (int n = 0; ok; ++n) {
        const int idx = item_of(n);
        if (n * (int)gridDim.x >= p.n_items) break;
        if (idx >= p.n_items || !load_item(it, idx, p)) continue;
#pragma unroll
        for (int t = 0; t < QT; ++t) {
          if (it.n_kt[t] == 0 || !ok) continue;
          if (qn[t] > 0) ok = mbar_wait(q_free + t, (qn[t] - 1) & 1u, abort_flag, status, 61);
          if (!ok) continue;
          ++qn[t];
          mbar_expect_tx(q_ready + t, Q_BYTES);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            tma_load_2d(Qs + t * Q_BYTES + c * SUBQ, &q_map, q_ready + t, (p.head0 + it.h) * (DK + PR) + 64 * c,
                        it.s.q_begin + it.row0 + t * ROWS);
        }
        const int row = it.base + it.k_begin - it.s.k_first;
        for (int j = 0; j <= it.n_tiles && ok; ++j) {
          if (j < it.n_tiles) {
            const uint32_t st = kn % STAGES;
            ok = mbar_wait(k_empty + st, ((kn / STAGES) & 1u) ^ 1u, abort_flag, status, 62);
            if (!ok) break;
            mbar_expect_tx(k_full + st, K_BYTES);
            unsigned char* dst = Ks + st * K_BYTES;
            tma_load_2d(dst, &kv_map, k_full + st, it.h * (DK + DV), row + j * KT);
            tma_load_2d(dst + SUBK, &kv_map, k_full + st, it.h * (DK + DV) + 64, row + j * KT);
            tma_load_2d(dst + 2 * SUBK, &kr_map, k_full + st, 0, row + j * KT);
            ++kn;
          }
          if (j > 0) {                                   // K runs a tile ahead of V: its stages come free earlier
            const uint32_t st = vn % STAGES;
            ok = mbar_wait(v_empty + st, ((vn / STAGES) & 1u) ^ 1u, abort_flag, status, 63);
            if (!ok) break;
            mbar_expect_tx(v_full + st, V_BYTES);
            unsigned char* dst = Vs + st * V_BYTES;
            tma_load_2d(dst, &kv_map, v_full + st, it.h * (DK + DV) + DK, row + (j - 1) * KT);
            tma_load_2d(dst + SUBK, &kv_map, v_full + st, it.h * (DK + DV) + DK + 64, row + (j - 1) * KT);
            ++vn;
          }
        }
      }
      if (*abort_flag) {             // copies still in flight land before the block's shared memory is given up
        for (uint32_t i = kn > STAGES ? kn - STAGES : 0; i < kn; ++i)
          for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(k_full + i % STAGES, (i / STAGES) & 1u); ++t) __nanosleep(32);
        for (uint32_t i = vn > STAGES ? vn - STAGES : 0; i < vn; ++i)
          for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(v_full + i % STAGES, (i / STAGES) & 1u); ++t) __nanosleep(32);
        for (int tt = 0; tt < QT; ++tt)
          for (uint32_t t = 0; qn[tt] > 0 && t < (1u << 16) && !mbar_try_wait(q_ready + tt, (qn[tt] - 1) & 1u); ++t) __nanosleep(32);
      }
    }
  } else if (warp == 1 || warp == MMA_WARP_1) {
    // ------------------------------------------------------------------ products, one thread per Q tile
    const int tt = warp == 1 ? 0 : 1;
    if (lane == 0) {
      const uint32_t id_s = instr_desc(KT), id_o = instr_desc(DV, true);
      const uint64_t qdesc = smem_desc(Qs + tt * Q_BYTES);
      uint32_t base_no = 0, sq = 0, n_mine = 0;
      bool ok = true;
      for (int n = 0; ok; ++n) {
        const int idx = item_of(n);
        if (n * (int)gridDim.x >= p.n_items) break;
        if (idx >= p.n_items || !load_item(it, idx, p)) continue;
        const int my_tiles = it.n_kt[tt], n_tiles = it.n_tiles;
        if (my_tiles > 0) ok = mbar_wait(q_ready + tt, n_mine & 1u, abort_flag, status, 64);
        tc_fence_after();
        auto issue_s = [&](int j) -> bool {
          const uint32_t kn = base_no + (uint32_t)j, bf = (sq + (uint32_t)j) & 1u, st = kn % STAGES;
          if (!mbar_wait(k_full + st, (kn / STAGES) & 1u, abort_flag, status, 65)) return false;
          // (the buffer's last user announced its P, which this thread has seen, after it had read S)
          tc_fence_after();
          const uint64_t kdesc = smem_desc(Ks + st * K_BYTES);
          const uint32_t d = tmem + (uint32_t)(tt * 128) + bf * 64u;
#pragma unroll
          for (int ks = 0; ks < (DK + PR) / 16; ++ks) {
            const uint64_t a_off = (uint64_t)((ks >> 2) * (SUBQ >> 4) + 2 * (ks & 3));
            const uint64_t b_off = (uint64_t)((ks >> 2) * (SUBK >> 4) + 2 * (ks & 3));
            tc_mma(d, qdesc + a_off, kdesc + b_off, id_s, ks > 0 ? 1u : 0u);
          }
          tc_commit(s_full + 2 * tt + bf);
          tc_commit(k_empty + st);
          if (j == my_tiles - 1) tc_commit(q_free + tt);
          return true;
        };
        for (int j = 0; j < 2 && j < my_tiles && ok; ++j) ok = issue_s(j);
        for (int j = 0; j < n_tiles && ok; ++j) {
          const uint32_t kn = base_no + (uint32_t)j, st = kn % STAGES;
          if (j >= my_tiles) {
            // tiles that only the other Q tile sees: this one's share of their release, once they have arrived
            ok = mbar_wait(k_full + st, (kn / STAGES) & 1u, abort_flag, status, 65);
            if (ok) mbar_arrive(k_empty + st);
            if (ok) ok = mbar_wait(v_full + st, (kn / STAGES) & 1u, abort_flag, status, 66);
            if (ok) mbar_arrive(v_empty + st);
            continue;
          }
          const uint32_t pn = sq + (uint32_t)j, bf = pn & 1u;
          ok = mbar_wait(p_ready + 2 * tt + bf, (pn >> 1) & 1u, abort_flag, status, 67);
          if (ok) ok = mbar_wait(v_full + st, (kn / STAGES) & 1u, abort_flag, status, 66);
          if (ok && j == 0 && n_mine > 0) ok = mbar_wait(o_free + tt, (n_mine - 1) & 1u, abort_flag, status, 68);
          if (!ok) break;
          tc_fence_after();
          const uint32_t p_tmem = tmem + (uint32_t)(tt * 128) + bf * 64u;
          const uint64_t vdesc = desc_mnmajor(Vs + st * V_BYTES, SUBK);
          const uint32_t d = tmem + (uint32_t)(256 + tt * 128);
#pragma unroll
          for (int part = 1; part >= 0; --part)                       // the remainders, then the rounded weights
#pragma unroll
            for (int kk = 0; kk < KT / 16; ++kk)
              tc_mma_a_tmem(d, p_tmem + (uint32_t)(32 * part + 8 * kk), vdesc + (uint64_t)(kk * ((16 * 128) >> 4)), id_o,
                            (j > 0 || part == 0 || kk > 0) ? 1u : 0u);
          tc_commit(pv_done + 2 * tt + bf);
          tc_commit(v_empty + st);
          if (j + 2 < my_tiles) ok = issue_s(j + 2);
        }
        base_no += (uint32_t)n_tiles;
        sq += (uint32_t)my_tiles;
        n_mine += my_tiles > 0 ? 1u : 0u;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, one thread per row
    const int tt = (warp - 2) >> 2, quad = warp & 3, row = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const uint32_t tmem_o = tmem + (uint32_t)(256 + tt * 128) + lane_addr;
    uint32_t sq = 0;
    bool ok = true;
    for (int n = 0; ok; ++n) {
      const int idx = item_of(n);
      if (n * (int)gridDim.x >= p.n_items) break;
      if (idx >= p.n_items || !load_item(it, idx, p)) continue;
      const int my_tiles = it.n_kt[tt];
      if (my_tiles == 0) continue;
      const int qi = it.row0 + tt * ROWS + row;
      const bool live = qi < it.s.q_len;
      const int lim = live ? it.s.pos0 + qi : -1;
      const int lo = live ? bspec::mask_lo(it.s.pos0 + qi, p.window) : 0;
      const int my_k_end = it.k_end_t[tt];
      // m_ref follows the running maximum lazily: it is looked for again when a tile's weights sum to more than 2^14, and
      // O and l are rescaled if it has grown by more than 8
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < my_tiles && ok; ++j) {
        const uint32_t no = sq + (uint32_t)j, b = no & 1u;
        ok = mbar_wait(s_full + 2 * tt + b, (no >> 1) & 1u, abort_flag, status, 69);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const int key0 = it.k_begin + j * KT;
        const bool need_mask = key0 + KT - 1 > lim || key0 < lo || key0 + KT > my_k_end;
        uint32_t sv[2][32];
        const uint32_t s_addr = tmem + (uint32_t)(tt * 128) + b * 64u + lane_addr;
        tc_ld32(s_addr, sv[0]);
        tc_ld32(s_addr + 32u, sv[1]);
        tc_wait_ld();
        // weights 2^(scale S - m) of the row, their two parts back into tensor memory, their sum returned
        auto exponentials = [&](float neg_m) -> float {
          const uint64_t scale2 = pack2(p.scale_log2, p.scale_log2), neg_m2 = pack2(neg_m, neg_m);
          uint64_t l2[2] = {0ull, 0ull};
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t hi[16], rest[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              float p0, p1;
              unpack2(fma2(pack2(__uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1])), scale2, neg_m2), p0, p1);
              p0 = ex2(p0);
              p1 = ex2(p1);
              l2[(i >> 1) & 1] = add2(l2[(i >> 1) & 1], pack2(p0, p1));
              const __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);
              const uint32_t h = *reinterpret_cast<const uint32_t*>(&hh);
              hi[i >> 1] = h;
              const __nv_bfloat162 rr = __floats2bfloat162_rn(p0 - __uint_as_float(h << 16), p1 - __uint_as_float(h & 0xffff0000u));
              rest[i >> 1] = *reinterpret_cast<const uint32_t*>(&rr);
            }
            tc_st16(s_addr + 16u * c, hi);
            tc_st16(s_addr + 32u + 16u * c, rest);
          }
          float la, lb;
          unpack2(add2(l2[0], l2[1]), la, lb);
          return la + lb;
        };
        float corr = 1.f, row_sum = 0.f;
        bool full_path = __any_sync(0xffffffffu, need_mask || m_ref == -INFINITY);
        if (!full_path) {
          row_sum = exponentials(-m_ref);
          full_path = __any_sync(0xffffffffu, !(row_sum <= 16384.f));
          if (full_path) tc_wait_st();                 // those stores land before the ones that replace them
        }
        if (full_path) {
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
          if (need_mask) {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const int key = key0 + 32 * c + i;
                if (!(key <= lim && key >= lo && key < my_k_end)) sv[c][i] = 0xff800000u;
                mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sv[c][i]));
              }
          } else {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; i += 2)
                mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1]));
          }
          const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
          if (mx > m_ref + 8.f || m_ref == -INFINITY) {
            const float m_new = fmaxf(m_ref, mx);
            corr = m_new == -INFINITY ? 1.f : ex2(m_ref - m_new);
            m_ref = m_new;
            l *= corr;
          }
          __syncwarp();
          row_sum = exponentials(m_ref == -INFINITY ? 0.f : -m_ref);
        }
        l += row_sum;
        if (j >= 1 && __any_sync(0xffffffffu, corr != 1.f)) {
          ok = mbar_wait(pv_done + 2 * tt + (b ^ 1u), ((no - 1) >> 1) & 1u, abort_flag, status, 70);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < DV / 32; ++c) {
            uint32_t v[32];
            tc_ld32(tmem_o + 32u * c, v);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * corr);
            tc_st32(tmem_o + 32u * c, v);
          }
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready + 2 * tt + b);
      }
      const uint32_t n_last = sq + (uint32_t)my_tiles - 1u;
      if (ok) ok = mbar_wait(pv_done + 2 * tt + (n_last & 1u), (n_last >> 1) & 1u, abort_flag, status, 71);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      if (ok) {
        float l_all = l;
        if (p.sink != nullptr && l > 0.f) l_all += ex2(p.sink[p.head0 + it.h] * 1.4426950408889634f - m_ref);
        const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
        uint4* dst = reinterpret_cast<uint4*>(p.out + (long long)(it.s.q_begin + qi) * p.o_row + (long long)(p.head0 + it.h) * p.o_head);
#pragma unroll
        for (int c = 0; c < DV / 32; ++c) {
          uint32_t v[32];
          tc_ld32(tmem_o + 32u * c, v);
          tc_wait_ld();
          if (c == DV / 32 - 1) {                      // O is in registers: the next item's first P V may replace it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free + tt);
          }
          if (live) {
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) {
              uint32_t w[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(v[8 * k4 + 2 * i]) * inv, __uint_as_float(v[8 * k4 + 2 * i + 1]) * inv);
                w[i] = *reinterpret_cast<const uint32_t*>(&hh);
              }
              dst[4 * c + k4] = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      }
      sq += (uint32_t)my_tiles;
    }
  }
  bspec::pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}
}  // namespace

// 1 if the sizes are the ones these kernels are made for.
BSPEC_API int bspec_latent_prompt_supported(int R, int dim, int rot_dim, int vdim) {
  return dim == DK && rot_dim == PR && vdim == DV && R > 0 && R % 8 == 0 ? 1 : 0;
}

// The entries that the portions of at least ``min_q`` tokens see, out of their pages: cbuf [T, R], krbuf [T, 64], and
// base [n_entries], the first row of each.  T: the sum over those portions of their keys' number (from the first key the
// window leaves their first token, down to a multiple of 64) rounded up to 64.
BSPEC_API int bspec_latent_gather(const void* cache, const int* qo_indptr, const int* positions, const int* kv_indptr,
                                  const int* kv_indices, int n_entries, int R, int page_size, int window, int min_q, int T,
                                  void* cbuf, void* krbuf, int* base, long long n_pages, cudaStream_t stream) {
  if (n_entries <= 0 || T <= 0) return 0;
  if (R % 8 != 0 || T % KT != 0 || window < 0) return (int)cudaErrorInvalidValue;
  BSPEC_LAUNCH(latent_gather_kernel, dim3(T / KT), 256, 0, stream, (const __nv_bfloat16*)cache, qo_indptr, positions, kv_indptr,
               kv_indices, n_entries, R, page_size, window, min_q, (__nv_bfloat16*)cbuf, (__nv_bfloat16*)krbuf, base, n_pages);
  return BSPEC_LAUNCH_CHECK();
}

// Attention of the portions of at least ``min_q`` tokens over heads head0 .. head0 + heads - 1.  q: [n, H (dim + rot)] with
// the rotated parts rotated; kv [T, heads (dim + vdim)]: keys and values of those heads; out: written at token * o_row +
// head * o_head, 16-byte aligned rows; sink: float32 per head or null; max_q: the longest portion.
BSPEC_API int bspec_latent_prompt(const void* q, long long q_row, int n_tokens, int H, const void* kv, const void* krbuf,
                                  const int* base, int T, void* out, long long o_row, long long o_head, const int* qo_indptr,
                                  const int* positions, int n_entries, int max_q, int head0, int heads, int window, int min_q,
                                  float scale, const float* sink, int* status, cudaStream_t stream) {
  if (n_entries <= 0 || T <= 0 || heads <= 0) return 0;
  if (!(scale > 0.f) || window < 0 || q_row % 8 != 0 || ((uintptr_t)q & 15) || ((uintptr_t)out & 15) || o_row % 8 != 0 || o_head % 8 != 0)
    return (int)cudaErrorInvalidValue;
  auto fn = encode_fn();
  if (fn == nullptr) return (int)cudaErrorInvalidValue;
  CUtensorMap q_map, kv_map, kr_map;
  auto make = [&](CUtensorMap* map, const void* base_, long long rows, long long cols, long long ld, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64u, (cuuint32_t)box_rows}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base_), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  const long long kv_cols = (long long)heads * (DK + DV);
  if (!make(&q_map, q, n_tokens, (long long)H * (DK + PR), q_row, ROWS) || !make(&kv_map, kv, T, kv_cols, kv_cols, KT) ||
      !make(&kr_map, krbuf, T, PR, PR, KT))
    return (int)cudaErrorInvalidValue;
  static bool set[bspec::kMaxDevices] = {};
  bool& done = set[bspec::current_device()];
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(latent_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const long long n_items = (long long)((max_q + QT * ROWS - 1) / (QT * ROWS)) * heads * n_entries;
  if (n_items > (1ll << 30)) return (int)cudaErrorInvalidConfiguration;
  Params p;
  p.out = (__nv_bfloat16*)out;
  p.o_row = o_row;
  p.o_head = o_head;
  p.qo_indptr = qo_indptr;
  p.positions = positions;
  p.base = base;
  p.sink = sink;
  p.status = status;
  p.n_entries = n_entries;
  p.n_items = (int)n_items;
  p.head0 = head0;
  p.heads = heads;
  p.window = window;
  p.min_q = min_q;
  p.scale_log2 = scale * 1.4426950408889634f;
  BSPEC_LAUNCH(latent_prompt_kernel, dim3((unsigned)min(n_items, (long long)bspec::sm_count())), THREADS, SMEM, stream, q_map, kv_map,
               kr_map, p);
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_DEFINE_TRACE_SETTER(bspec_trace_set_latent_prompt)
BSPEC_DEFINE_BOUNDS_REPORT(bspec_bounds_report_latent_prompt)
