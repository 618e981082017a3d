// Latent attention in bfloat16 on the tensor cores (mma.sync m16n8k16, float32 accumulation), prompt portions and
// decoded tokens alike.  All heads of a request read the same cache entries [c | kr] (R + P numbers), so the rows
// of a tile are (token, head) pairs: row = token * H + head, 16 * RG rows per CTA (RG row groups of 16: 64 rows for
// prompt portions, 16 or 32 for decoded tokens of models with up to 16 or 32 heads), and one pass over the request's
// entries serves every head.  A CTA is RG x CH warps: warp (rg, ch) owns 16 rows, 32 / CH keys of every score tile
// and R / CH columns of the output.  Per tile of 32 entries:
//
//   S = Q K^T over all R + P numbers (the entry is the key), scaled, causal mask, to shared memory in float32;
//   online softmax in float32, four threads per row; the weights are left as TWO bfloat16 numbers, the rounded
//   weight and the rounding's remainder, so that the product with the values carries them to 2^-17;
//   O += P_hi V + P_lo V with V the first R numbers of the same tile.
// The warps of a row group meet at a barrier of their own between these phases (the row groups drift apart, so
// one's softmax runs under another's products); the whole CTA meets once per tile, when the next tile has landed.
//
// Entries arrive by cp.async; the block-table lookup of a tile is made one tile before its copies.  A CTA holds
// two tiles of entries (the next one arrives under the current one's products: the 64-row tiles) or one (32-row
// tiles of prompt portions and the 16- and 32-row tiles of decoded tokens: two to four CTAs then share an SM and
// cover each other's loads, which measured faster).  In steps of few rows and many entries (decode) the requests' key
// tiles are dealt to the CTAs in even shares (``deal``); a CTA leaves (max, sum, unnormalised output) of its share for the
// join kernel, which adds a request's shares in their order.
#include "common.cuh"
#include <math.h>
#include <stdlib.h>
using namespace bspec;

namespace {

constexpr int BN = 32;

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
// ldmatrix on 32-bit shared-space addresses (formed once per kernel, advanced by byte offsets)
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm_x2(uint32_t (&r)[2], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n"
               : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ``shares``: score tiles in shared memory, 1 or (kernels that divide the numbers of an entry) one per warp of a row group.
__host__ __device__ inline size_t smem_bytes(int D, int BM, int stages = 2, int shares = 1) {
  const int DP = D + 8;
  return (size_t)(BM + stages * BN) * DP * 2 + (size_t)shares * BM * (BN + 8) * 4 + 2 * (size_t)BM * (BN + 8) * 2 + 3 * BM * 4;
}

// The work of a step of few rows, dealt evenly: the requests' key tiles are cut into shares of ``per`` tiles, as many in all as CTAs
// fit the device at once (a request has at least one, at most MAX_SHARES), and CTA z takes the z-th.  Every CTA finds that out
// for itself from the lengths, so a captured step follows them.  ``per`` is the least of TRY lengths from the even share up, each up
// to a sixteenth longer than the one before (then a quarter of the even share), whose shares all fit: a request's last share is
// shorter than the others, and a share more than fit runs after all others.  64 requests of 300 to
// 4,096 entries, 16 heads: 100 us with as many shares for each as for the longest, 55 dealt; requests of one length lose nothing
// by it: 64 of 4,096 entries 117 / 111 (141 where a few shares ran in a second wave), 64 of 1,000 43 / 41 (57), 256 of 300, a
// share each, 54 / 54 (73).  At latents of 128 and 256 the dealing itself shows, 256 of 300 26 / 29.  Shares of at least two tiles: a
// captured step whose bound is 4,608 entries, 5 requests of 100 16.6 us (of four tiles, all in one share, 20.2), 2 of 2,000 23.7 (of
// one tile, 40 shares to join, 28.9).
constexpr int MAX_SHARES = 64, MIN_TILES = 2, TRY = 16, OWN = 4;
struct Share {
  int e, split, first, count, per;       // request (-1: none), which of its shares, its first share and how many it has
};
template <int NT>
__device__ __forceinline__ Share deal(int z, const int* __restrict__ qo_indptr, const int* __restrict__ positions, int n_entries,
                                      int window, int skip_from, int want_shares) {
  __shared__ int part[3][NT / 32], tried[TRY][NT / 32], found[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto tiles_of = [&](int e) -> int {
    if (e >= n_entries) return 0;
    const int q0 = qo_indptr[e], q1 = qo_indptr[e + 1];
    if (q1 <= q0 || q1 - q0 >= skip_from) return 0;
    const int pos0 = positions[q0];
    return (pos0 + q1 - q0 - 1) / BN + 1 - (window > 0 ? max(0, pos0 - window + 1) / BN : 0);
  };
  if (tid == 0) found[0] = -1;
  int own[OWN];                                    // this thread's requests among the first NT * OWN, asked for at once
#pragma unroll
  for (int k = 0; k < OWN; ++k) own[k] = tiles_of(tid * OWN + k);
  auto each = [&](auto visit) {                    // visit(this thread's first request, its OWN requests' tiles), for all requests
    visit(tid * OWN, own);
    for (int e0 = NT * OWN; e0 < n_entries; e0 += NT * OWN) {
      int more[OWN];
#pragma unroll
      for (int k = 0; k < OWN; ++k) more[k] = tiles_of(e0 + tid * OWN + k);
      visit(e0 + tid * OWN, more);
    }
  };
  int total = 0, most = 0;
  each([&](int, const int (&t)[OWN]) {
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      total += t[k];
      most = max(most, t[k]);
    }
  });
  total = __reduce_add_sync(0xffffffffu, total);
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) {
    part[0][warp] = total;
    part[1][warp] = most;
  }
  __syncthreads();
  total = most = 0;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) {
    total += part[0][w];
    most = max(most, part[1][w]);
  }
  const int even = max(MIN_TILES, max((total + want_shares - 1) / want_shares, (most + MAX_SHARES - 1) / MAX_SHARES));
  auto length = [&](int i) -> int { return even + (i <= 8 ? (even * i + 15) / 16 : (even * (i - 6) + 3) / 4); };
  int per = even;
  if (n_entries <= want_shares) {                  // (else in waves)
    int shares[TRY];
    float inverse[TRY];                              // (a share more or less by rounding only moves the choice)
#pragma unroll
    for (int i = 0; i < TRY; ++i) {
      shares[i] = 0;
      inverse[i] = __fdividef(1.f, (float)length(i));
    }
    each([&](int, const int (&t)[OWN]) {
#pragma unroll
      for (int k = 0; k < OWN; ++k)
        if (t[k] > 0)
#pragma unroll
          for (int i = 0; i < TRY; ++i) shares[i] += __float2int_ru((float)t[k] * inverse[i] - 1e-3f);
    });
#pragma unroll
    for (int i = 0; i < TRY; ++i) {
      const int sum = __reduce_add_sync(0xffffffffu, shares[i]);
      if (lane == i) tried[i][warp] = sum;
    }
    __syncthreads();
    bool fits = false;
    if (lane < TRY) {
      int sum = 0;
#pragma unroll
      for (int w = 0; w < NT / 32; ++w) sum += tried[lane][w];
      fits = sum <= want_shares;
    }
    const unsigned first_fit = __ballot_sync(0xffffffffu, fits);
    if (first_fit != 0) per = length(__ffs(first_fit) - 1);
  }
  int before = 0;
  each([&](int e, const int (&t)[OWN]) {
    int n[OWN], mine = 0;
#pragma unroll
    for (int k = 0; k < OWN; ++k) mine += n[k] = (t[k] + per - 1) / per;
    int sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    if (lane == 31) part[2][warp] = sum;
    __syncthreads();
    int first = before + sum - mine;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
      if (w < warp) first += part[2][w];
      before += part[2][w];
    }
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      if (z >= first && z < first + n[k]) {
        found[0] = e + k;
        found[1] = first;
        found[2] = n[k];
      }
      first += n[k];
    }
    __syncthreads();
  });
  Share s;
  s.e = found[0];
  s.first = found[1];
  s.count = found[2];
  s.split = z - found[1];
  s.per = per;
  return s;
}

// RG row groups x CH column groups of warps; NT: n-tiles (of 8 columns) of the output one warp may own,
// R / (8 CH) <= NT.
// ST: tiles of entries in shared memory: 2 (the next one arrives under the current one's products) or 1 (two CTAs
// share an SM instead and cover each other's loads).
// DS: the CH warps of a row group divide the numbers of an entry between them instead of the keys.  A warp then multiplies
// all 32 keys of the tile with a CH-th of the R + P numbers, 3 fragment loads for 4 products instead of 2 for 1, and leaves
// a share of the scores that the softmax adds up in the warps' order.
template <int RG, int CH, int NT, int ST = 2, bool DS = false>
__global__ void __launch_bounds__(32 * RG * CH)
latent_attn_mma_kernel(const __nv_bfloat16* __restrict__ ql, long long ql_row, long long ql_head,
                       const __nv_bfloat16* __restrict__ qr, long long qr_row, long long qr_head,
                       __nv_bfloat16* __restrict__ out, long long o_row, long long o_head,
                       const __nv_bfloat16* __restrict__ cache, const int* __restrict__ qo_indptr,
                       const int* __restrict__ positions, const int* __restrict__ kv_indptr,
                       const int* __restrict__ kv_indices, int H, int R, int P, int page_size, float scale,
                       float* __restrict__ o_part, float* __restrict__ ml_part, long long n_pages,
                       const float* __restrict__ inv_freq, float magnitude, int window,
                       const float* __restrict__ sink, int skip_from, int* __restrict__ plan, int n_entries,
                       int rows_max, int want_shares) {
  constexpr int BM = 16 * RG;
  constexpr int KW = BN / CH;                     // keys of a score tile per warp: 16 or 8
  constexpr int TPR = 2 * CH, KPT = BN / TPR;     // softmax: threads per row, keys per thread
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // (the step's lengths were uploaded before its first kernel: they may be read before the wait)
  Share mine = {(int)blockIdx.y, 0, 0, 0, 0};
  if (plan != nullptr) mine = deal<32 * RG * CH>(blockIdx.z, qo_indptr, positions, n_entries, window, skip_from, want_shares);
  bspec::pdl_prologue(43);
  if (mine.e < 0) return;
  const int D = R + P, DP = D + 8;
  constexpr int PP = BN + 8, SP = BN + 8;
  __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __nv_bfloat16* Ks = Qs + (size_t)BM * DP;
  float* Ss = reinterpret_cast<float*>(Ks + (size_t)ST * BN * DP);
  __nv_bfloat16* Ph = reinterpret_cast<__nv_bfloat16*>(Ss + (size_t)(DS ? CH : 1) * BM * SP);
  __nv_bfloat16* Pl = Ph + (size_t)BM * PP;
  float* row_m = reinterpret_cast<float*>(Pl + (size_t)BM * PP);
  float* row_l = row_m + BM;
  float* row_c = row_l + BM;

  const int e = mine.e, split = mine.split;
  const int q_begin = qo_indptr[e], q_len = qo_indptr[e + 1] - q_begin;
  if (plan != nullptr && split == 0 && blockIdx.x == 0)                            // for the join
    for (int t = threadIdx.x; t < q_len; t += 32 * RG * CH)
      *reinterpret_cast<int2*>(plan + 2 * (q_begin + t)) = make_int2(mine.first * rows_max + t * H, mine.count);
  if (q_len >= skip_from) return;                  // another kernel's portions
  const long long rows_total = (long long)q_len * H;
  const long long row0 = (long long)blockIdx.x * BM;
  if (row0 >= rows_total) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rg = warp % RG, ch = warp / RG;
  const int pos0 = positions[q_begin];
  const int last_tok = (int)min((long long)q_len - 1, (row0 + BM - 1) / H);
  const int max_pos = pos0 + last_tok;
  // with a window the CTA's first row sees nothing before min_key: the tiles start there, and entries before it
  // (their pages may have been given back) are never looked up
  const int min_key = window > 0 ? max(0, pos0 + (int)(row0 / H) - window + 1) : 0;
  const int tile0 = min_key / BN;
  const int n_tiles = max_pos / BN + 1;
  const int per = plan != nullptr ? mine.per : n_tiles - tile0;
  const int from = plan != nullptr ? (window > 0 ? max(0, pos0 - window + 1) / BN : 0) : tile0;      // the shares' first tile
  const int t_begin = max(tile0, from + split * per), t_end = min(n_tiles, from + (split + 1) * per);
  const int* table = kv_indices + kv_indptr[e];

  // ---- queries: row r holds [ql | qr] of (token, head) = divmod(row0 + r, H); rows past the portion are zero.
  // With a frequency table the rotated part arrives unrotated and is rotated here (adjacent pairs, the angle in
  // float64 from the two-float frequencies, cosine and sine times the magnitude), then rounded as a separate
  // rotation kernel would have left it.
  for (int r = warp; r < BM; r += RG * CH) {      // a warp per row: its token and head are found once
    const long long row = row0 + r;
    const bool live = row < rows_total;
    const int tq = live ? (int)((unsigned)row / (unsigned)H) : 0;          // rows_total fits 32 bits (checked at launch)
    const int h = live ? (int)((unsigned)row - (unsigned)tq * (unsigned)H) : 0;
    const long long t = q_begin + tq;
    const __nv_bfloat16* src_l = ql + t * ql_row + h * ql_head;
    const __nv_bfloat16* src_r = qr + t * qr_row + h * qr_head;
    __nv_bfloat16* dst = Qs + (size_t)r * DP;
    for (int d = 2 * lane; d < R; d += 64) {
      const float u = live ? __bfloat162float(src_l[d]) : 0.f, v = live ? __bfloat162float(src_l[d + 1]) : 0.f;
      *reinterpret_cast<__nv_bfloat162*>(dst + d) = __floats2bfloat162_rn(u, v);
    }
    const int pos = live ? positions[t] : 0;
    for (int d = 2 * lane; d < P; d += 64) {
      float u = live ? __bfloat162float(src_r[d]) : 0.f, v = live ? __bfloat162float(src_r[d + 1]) : 0.f;
      if (inv_freq != nullptr && live) {
        const int j = d / 2, half = P / 2;
        const double f = (double)inv_freq[j] + (double)inv_freq[half + j];
        double ang = (double)pos * f;
        ang -= 6.283185307179586476925286766559 * rint(ang * 0.15915494309189533576888376337251);
        float sn, cs;
        sincosf((float)ang, &sn, &cs);
        sn *= magnitude;
        cs *= magnitude;
        const float ru = u * cs - v * sn, rv = v * cs + u * sn;
        u = ru;
        v = rv;
      }
      *reinterpret_cast<__nv_bfloat162*>(dst + R + d) = __floats2bfloat162_rn(u, v);
    }
  }
  if (tid < BM) {
    row_m[tid] = -INFINITY;
    row_l[tid] = 0.f;
  }

  // A tile's entries are dealt to the warps, one entry at a time; the lanes copy its 16-byte pieces.  The page
  // of an entry is looked up once per entry (a shift when the page size is a power of two).
  const int chunks = D / 8;                       // 16-byte pieces of an entry
  const int ps_shift = (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;
  // Lane j of a warp looks up the page of the warp's j-th entry of a tile; the lookup for a tile is made one
  // tile ahead of its copies, so that its latency passes under the products in between.
  constexpr int NW = RG * CH, KPW = BN / NW;      // warps; entries of a tile per warp
  auto lookup = [&](int tile) -> long long {      // element offset of the lane's entry in the cache, -1: none
    long long off = -1;
    if (lane < KPW && tile < t_end) {
      const int key = tile * BN + warp + lane * NW;
      if (key <= max_pos && key >= min_key) {
        const int slot = ps_shift >= 0 ? key >> ps_shift : key / page_size;
        const int page = table[slot];
        if (bspec::in_range(page, n_pages, 112)) off = ((long long)page * page_size + (key - slot * page_size)) * D;
      }
    }
    return off;
  };
  auto load_tile = [&](int buf, long long mine) {
    __nv_bfloat16* dst = Ks + (size_t)buf * BN * DP;
#pragma unroll
    for (int j = 0; j < KPW; ++j) {
      const long long off = __shfl_sync(0xffffffffu, mine, j);
      const bool valid = off >= 0;
      const __nv_bfloat16* src = cache + (valid ? off : 0);
      __nv_bfloat16* d = dst + (size_t)(warp + j * NW) * DP;
      for (int part = lane; part < chunks; part += 32) cp_async16(d + part * 8, src + (valid ? part * 8 : 0), valid);
    }
  };
  auto group_barrier = [&]() {
    if (RG == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + rg), "r"(32 * CH) : "memory");
  };

  float o[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  const int ntw = R / (8 * CH);                   // n-tiles this warp owns
  const int col0 = ch * (R / CH);                 // its first output column
  const int mat = lane >> 3, r8 = lane & 7;
  const int qrow = lane >> 2, qcol = 2 * (lane & 3);
  // this thread's softmax row: the row group's 32 CH threads, TPR per row
  const int tg = ch * 32 + lane;
  const int srow = 16 * rg + tg / TPR, spart = tg % TPR;
  // this lane's ldmatrix addresses (shared space, bytes): its row of the query fragments, of a key tile's score
  // fragments, of the weight fragments, and of the value fragments (transposed loads)
  const uint32_t qa_s = smem_addr(Qs + (size_t)(16 * rg + 8 * (mat & 1) + r8) * DP + 8 * (mat >> 1));
  const uint32_t kb_s = KW == 16 ? smem_addr(Ks + (size_t)(KW * ch + 8 * (mat >> 1) + r8) * DP + 8 * (mat & 1))
                                 : smem_addr(Ks + (size_t)(KW * ch + r8) * DP + 8 * (mat & 1));
  // DS: both halves of the tile's keys, 16 rows apart
  const uint32_t kd_s = smem_addr(Ks + (size_t)(8 * (mat >> 1) + r8) * DP + 8 * (mat & 1));
  const uint32_t ph_s = smem_addr(Ph + (size_t)(16 * rg + 8 * (mat & 1) + r8) * PP + 8 * (mat >> 1));
  const uint32_t pl_s = smem_addr(Pl + (size_t)(16 * rg + 8 * (mat & 1) + r8) * PP + 8 * (mat >> 1));
  const uint32_t vt_s = smem_addr(Ks + (size_t)(8 * (mat & 1) + r8) * DP + col0 + 8 * (mat >> 1));
  // the last key each of this thread's two score rows may see (-1: the row is past the portion)
  int row_pos[2], row_lo[2];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const long long row = row0 + 16 * rg + qrow + 8 * half;
    row_pos[half] = row < rows_total ? pos0 + (int)(row / H) : -1;
    row_lo[half] = window > 0 ? row_pos[half] - window + 1 : 0;         // the first key the row sees
  }

  // the same for this thread's softmax row
  const long long soft_row = row0 + srow;
  const int soft_pos = soft_row < rows_total ? pos0 + (int)(soft_row / H) : -1;
  const int soft_lo = window > 0 ? soft_pos - window + 1 : 0;

  long long ahead = lookup(t_begin);
  if (t_begin < t_end) load_tile(0, ahead);
  cp_async_commit();
  ahead = lookup(t_begin + 1);
  for (int tile = t_begin; tile < t_end; ++tile) {
    const int buf = ST == 2 ? (tile - t_begin) & 1 : 0;
    cp_async_wait<0>();
    __syncthreads();                              // the tile is here, and everybody is done with the tile before
    if (ST == 2) {
      if (tile + 1 < t_end) load_tile(buf ^ 1, ahead);
      cp_async_commit();
      ahead = lookup(tile + 2);
    }
    if constexpr (DS) {
      // ---- S: this warp's 16 rows x 32 keys over its share of the numbers, fragments fetched one k step ahead
      float s[4][4];
#pragma unroll
      for (int y = 0; y < 4; ++y) s[y][0] = s[y][1] = s[y][2] = s[y][3] = 0.f;
      const uint32_t kb = kd_s + (uint32_t)buf * (uint32_t)(BN * DP * 2);
      const int nks = D / 16, k_begin = nks * ch / CH, k_end = nks * (ch + 1) / CH;
      uint32_t fa[2][4], f0[2][4], f1[2][4];
      auto fetch = [&](int slot, int k) {
        ldsm_x4(fa[slot], qa_s + 32u * k);
        ldsm_x4(f0[slot], kb + 32u * k);
        ldsm_x4(f1[slot], kb + 32u * k + (uint32_t)(16 * DP * 2));
      };
      auto mul = [&](int slot) {
        mma_bf16(s[0], fa[slot], f0[slot][0], f0[slot][1]);
        mma_bf16(s[1], fa[slot], f0[slot][2], f0[slot][3]);
        mma_bf16(s[2], fa[slot], f1[slot][0], f1[slot][1]);
        mma_bf16(s[3], fa[slot], f1[slot][2], f1[slot][3]);
      };
      if (k_begin < k_end) fetch(0, k_begin);
      int k = k_begin;
      for (; k + 2 <= k_end; k += 2) {
        fetch(1, k + 1);
        mul(0);
        if (k + 2 < k_end) fetch(0, k + 2);
        mul(1);
      }
      if (k < k_end) mul(0);
      float* share = Ss + (size_t)ch * BM * SP;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half)
          *reinterpret_cast<float2*>(share + (16 * rg + qrow + 8 * half) * SP + 8 * nt + qcol) =
              make_float2(s[nt][2 * half], s[nt][2 * half + 1]);
    } else {
      // ---- S: this warp's 16 rows x KW keys, two accumulator sets over alternating k steps
      constexpr int NS = KW / 8;
      float s[4][NS][4];
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < NS; ++y) s[x][y][0] = s[x][y][1] = s[x][y][2] = s[x][y][3] = 0.f;
      const uint32_t kb = kb_s + (uint32_t)buf * (uint32_t)(BN * DP * 2);
      const int nks = D / 16;
      // The asm statements keep their order, so the loop is pipelined by hand: the fragments of k step i + 1 are
      // fetched before the products of step i are issued (two sets of fragment registers, four accumulator chains).
      uint32_t fa[2][4], fb[2][4];
      auto fetch = [&](int slot, uint32_t off) {                 // off: bytes along the row, 32 per k step
        ldsm_x4(fa[slot], qa_s + off);
        if (KW == 16) {
          ldsm_x4(fb[slot], kb + off);
        } else {
          uint32_t t[2];
          ldsm_x2(t, kb + off);
          fb[slot][0] = t[0];
          fb[slot][1] = t[1];
        }
      };
      auto mul = [&](float (&acc)[NS][4], int slot) {
        mma_bf16(acc[0], fa[slot], fb[slot][0], fb[slot][1]);
        if (KW == 16) mma_bf16(acc[NS - 1], fa[slot], fb[slot][2], fb[slot][3]);
      };
      fetch(0, 0u);
      int ks = 0;
      for (; ks + 4 <= nks; ks += 4) {
        fetch(1, 32u * (ks + 1));
        mul(s[0], 0);
        fetch(0, 32u * (ks + 2));
        mul(s[1], 1);
        fetch(1, 32u * (ks + 3));
        mul(s[2], 0);
        if (ks + 4 < nks) fetch(0, 32u * (ks + 4));
        mul(s[3], 1);
      }
      for (; ks < nks; ++ks) {
        mul(s[0], 0);
        if (ks + 1 < nks) fetch(0, 32u * (ks + 1));
      }
#pragma unroll
      for (int y = 0; y < NS; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          s[0][y][x] += s[1][y][x];
          s[2][y][x] += s[3][y][x];
        }
#pragma unroll
      for (int nt = 0; nt < NS; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int r = 16 * rg + qrow + 8 * half;
          const int c = KW * ch + 8 * nt + qcol;
          const int key = tile * BN + c;
          float2 v;
          v.x = (key <= row_pos[half] && key >= row_lo[half])
                    ? (s[0][nt][2 * half] + s[2][nt][2 * half]) * scale : -INFINITY;
          v.y = (key + 1 <= row_pos[half] && key + 1 >= row_lo[half])
                    ? (s[0][nt][2 * half + 1] + s[2][nt][2 * half + 1]) * scale : -INFINITY;
          *reinterpret_cast<float2*>(Ss + r * SP + c) = v;
        }
    }
    group_barrier();
    // ---- softmax: TPR threads per row, KPT keys each
    {
      float v[KPT];
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < KPT; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(Ss + srow * SP + KPT * spart + j);
        v[j] = x.x; v[j + 1] = x.y; v[j + 2] = x.z; v[j + 3] = x.w;
      }
      if constexpr (DS) {                          // the other shares, then scale and mask
#pragma unroll
        for (int w = 1; w < CH; ++w)
#pragma unroll
          for (int j = 0; j < KPT; j += 4) {
            const float4 x = *reinterpret_cast<const float4*>(Ss + (size_t)w * BM * SP + srow * SP + KPT * spart + j);
            v[j] += x.x; v[j + 1] += x.y; v[j + 2] += x.z; v[j + 3] += x.w;
          }
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
          const int key = tile * BN + KPT * spart + j;
          v[j] = key <= soft_pos && key >= soft_lo ? v[j] * scale : -INFINITY;
        }
      }
#pragma unroll
      for (int j = 0; j < KPT; ++j) mx = fmaxf(mx, v[j]);
#pragma unroll
      for (int x = 1; x < TPR; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      const float m_old = row_m[srow], l_old = row_l[srow];
      const float m_new = fmaxf(m_old, mx);
      float sum = 0.f;
      __align__(16) __nv_bfloat16 hi[KPT], lo[KPT];
#pragma unroll
      for (int j = 0; j < KPT; ++j) {
        const float p = m_new == -INFINITY ? 0.f : __expf(v[j] - m_new);
        sum += p;
        hi[j] = __float2bfloat16_rn(p);
        lo[j] = __float2bfloat16_rn(p - __bfloat162float(hi[j]));
      }
      if (KPT == 8) {
        *reinterpret_cast<uint4*>(Ph + srow * PP + KPT * spart) = *reinterpret_cast<const uint4*>(hi);
        *reinterpret_cast<uint4*>(Pl + srow * PP + KPT * spart) = *reinterpret_cast<const uint4*>(lo);
      } else {
        *reinterpret_cast<uint2*>(Ph + srow * PP + KPT * spart) = *reinterpret_cast<const uint2*>(hi);
        *reinterpret_cast<uint2*>(Pl + srow * PP + KPT * spart) = *reinterpret_cast<const uint2*>(lo);
      }
#pragma unroll
      for (int x = 1; x < TPR; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
      if (spart == 0) {
        const float corr = m_new == -INFINITY ? 1.f : __expf(m_old - m_new);
        row_m[srow] = m_new;
        row_l[srow] = l_old * corr + sum;
        row_c[srow] = corr;
      }
    }
    group_barrier();
    // ---- O = O * corr + P V over this warp's columns
    {
      const float c_lo = row_c[16 * rg + qrow], c_hi = row_c[16 * rg + qrow + 8];
      if (!__all_sync(0xffffffffu, c_lo == 1.f && c_hi == 1.f)) {      // some row's maximum moved
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          o[i][0] *= c_lo; o[i][1] *= c_lo; o[i][2] *= c_hi; o[i][3] *= c_hi;
        }
      }
      const uint32_t vt = vt_s + (uint32_t)buf * (uint32_t)(BN * DP * 2);
#pragma unroll
      for (int kk = 0; kk < BN / 16; ++kk) {
        uint32_t ah[4], al[4];
        ldsm_x4(ah, ph_s + 32 * kk);
        ldsm_x4(al, pl_s + 32 * kk);
        const uint32_t vk = vt + (uint32_t)kk * (uint32_t)(16 * DP * 2);
        uint32_t vb[2][4];                         // the value fragments, fetched one pair of tiles ahead
        ldsm_x4_trans(vb[0], vk);
#pragma unroll
        for (int nd = 0; nd < NT; nd += 2) {
          if (nd < ntw) {
            const int cur = (nd >> 1) & 1;
            if (nd + 2 < ntw) ldsm_x4_trans(vb[cur ^ 1], vk + 16 * (nd + 2));
            mma_bf16(o[nd], ah, vb[cur][0], vb[cur][1]);
            if (nd + 1 < ntw) mma_bf16(o[nd + 1], ah, vb[cur][2], vb[cur][3]);
            mma_bf16(o[nd], al, vb[cur][0], vb[cur][1]);
            if (nd + 1 < ntw) mma_bf16(o[nd + 1], al, vb[cur][2], vb[cur][3]);
          }
        }
      }
    }
    if (ST == 1) {                                // the one buffer is free once every warp has left the tile
      __syncthreads();
      if (tile + 1 < t_end) load_tile(0, ahead);
      cp_async_commit();
      ahead = lookup(tile + 2);
    }
  }
  cp_async_wait<0>();
  __syncthreads();          // row_m / row_l of the init (no tiles) or of the last tile, for every warp
  // The sink: a logit per head whose exponential joins the denominator.  The first share takes it, as one more
  // (valueless) key: its maximum, sum and output are rescaled the way a tile rescales them.
  if (sink != nullptr && split == 0) {
    if (tid < BM) {
      const long long row = row0 + tid;
      float corr = 1.f;
      if (row < rows_total) {
        const float sk = sink[(int)(row % H)];
        const float m_old = row_m[tid], m_new = fmaxf(m_old, sk);
        corr = m_old == -INFINITY ? 0.f : __expf(m_old - m_new);
        row_m[tid] = m_new;
        row_l[tid] = row_l[tid] * corr + __expf(sk - m_new);
      }
      row_c[tid] = corr;
    }
    __syncthreads();
    const float c_lo = row_c[16 * rg + qrow], c_hi = row_c[16 * rg + qrow + 8];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      o[i][0] *= c_lo; o[i][1] *= c_lo; o[i][2] *= c_hi; o[i][3] *= c_hi;
    }
  }

  // ---- results
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int r = 16 * rg + qrow + 8 * half;
    const long long row = row0 + r;
    if (row >= rows_total) continue;
    const long long t = q_begin + row / H;
    const int h = (int)(row % H);
    if (mine.count <= 1) {                         // the whole request is this CTA's
      const float inv = 1.f / row_l[r];
      __nv_bfloat16* op = out + t * o_row + h * o_head;
#pragma unroll
      for (int nd = 0; nd < NT; ++nd)
        if (nd < ntw) {
          const int c = col0 + 8 * nd + qcol;
          *reinterpret_cast<__nv_bfloat162*>(op + c) =
              __floats2bfloat162_rn(o[nd][2 * half] * inv, o[nd][2 * half + 1] * inv);
        }
    } else {
      const size_t slot = (size_t)(mine.first + split) * rows_max + (size_t)row;
      float* op = o_part + slot * R;
#pragma unroll
      for (int nd = 0; nd < NT; ++nd)
        if (nd < ntw) {
          const int c = col0 + 8 * nd + qcol;
          *reinterpret_cast<float2*>(op + c) = make_float2(o[nd][2 * half], o[nd][2 * half + 1]);
        }
      if (ch == 0 && (lane & 3) == 0) {
        ml_part[2 * slot] = row_m[r];
        ml_part[2 * slot + 1] = row_l[r];
      }
    }
  }
}

// out[row, :] = sum_s w_s O_s / sum_s w_s l_s with w_s = exp(m_s - max m), s ascending.  A block takes ``per_block`` (token, head)
// rows, one after the other, and goes on: the shares' weights are formed once (in parallel, into shared memory), then every
// thread adds its four columns, eight shares' numbers asked for at a time (one number each, four at a time: 0.5 us per share).
// Several rows where there are many: most then have a single share, and blocks that only see that took their launch's time (256
// requests of 128 heads: 17 us).
// ``plan``: per token the row of its first head in its request's first share and the number of shares, whose rows lie rows_max
// apart from share to share; a single share has left its result where it belongs, a portion of another kernel has none.
__global__ void __launch_bounds__(128)
latent_attn_join_kernel(const float* __restrict__ o_part, const float* __restrict__ ml_part, __nv_bfloat16* __restrict__ out,
                        long long o_row, long long o_head, int H, int R, const int* __restrict__ plan, int rows_max, int rows,
                        int per_block) {
  bspec::pdl_prologue(44);
  __shared__ float w[MAX_SHARES], l[MAX_SHARES];
  __shared__ float inv_l;
  for (int r0 = blockIdx.x * per_block; r0 < rows; r0 += gridDim.x * per_block)
    for (int r = r0; r < min(rows, r0 + per_block); ++r) {
      const int t = r / H, h = r - t * H;
      const int2 from = *reinterpret_cast<const int2*>(plan + 2 * t);
      const int n_shares = from.y;
      if (n_shares <= 1) continue;
      const size_t row = (size_t)from.x + h, step = rows_max;
      __syncthreads();                             // the row before is done with w
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const float2 none = make_float2(-INFINITY, 0.f);
        const float2* ml = reinterpret_cast<const float2*>(ml_part) + row;
        const float2 a = lane < n_shares ? ml[lane * step] : none, b = lane + 32 < n_shares ? ml[(lane + 32) * step] : none;
        const float M = warp_max(fmaxf(a.x, b.x));
        w[lane] = a.x == -INFINITY ? 0.f : expf(a.x - M);
        w[lane + 32] = b.x == -INFINITY ? 0.f : expf(b.x - M);
        l[lane] = a.y;
        l[lane + 32] = b.y;
        __syncwarp();
        if (lane == 0) {             // the sum in the order of the shares
          float L = 0.f;
#pragma unroll 8
          for (int s = 0; s < n_shares; ++s) {
            const float ws = w[s], ls = l[s];
            L = ws != 0.f ? fmaf(ws, ls, L) : L;
          }
          inv_l = 1.f / L;
        }
      }
      __syncthreads();
      const float inv = inv_l;
      for (int c = 4 * threadIdx.x; c < R; c += 512) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int s = 0; s < n_shares; ++s) {
          const float4 x = *reinterpret_cast<const float4*>(o_part + (row + s * step) * R + c);
          const float ws = w[s];
          if (ws != 0.f) acc.x = fmaf(ws, x.x, acc.x), acc.y = fmaf(ws, x.y, acc.y), acc.z = fmaf(ws, x.z, acc.z), acc.w = fmaf(ws, x.w, acc.w);
        }
        __nv_bfloat162* to = reinterpret_cast<__nv_bfloat162*>(out + t * o_row + h * o_head + c);
        to[0] = __floats2bfloat162_rn(acc.x * inv, acc.y * inv);
        to[1] = __floats2bfloat162_rn(acc.z * inv, acc.w * inv);
      }
    }
}

}  // namespace

// 1 if the tensor-core kernel takes these sizes (ranks and rotated part multiples of 16, latent at most 512,
// the tile fits shared memory), else 0.
BSPEC_API int bspec_latent_attention_mma_supported(int R, int P) {
  return (R > 0 && R % 16 == 0 && P >= 16 && P % 16 == 0 && R <= 512 && smem_bytes(R + P, 64) <= 220 * 1024) ? 1 : 0;
}

// How prompt portions are tiled: 2 (default) = 32 rows, 8 warps, one tile of entries, two CTAs per SM, when those
// fit (else as 0); 0 = 64 rows, 16 warps, two tiles of entries in flight; 1 = 64 rows, 8 warps.  Measured on a
// 4,096-token prompt with 16 / 32 heads, latent 512 + 64: 127 / 134, 118 / 126 and 110 / 116 TFLOP/s.  The
// environment variable is a tuning switch.
static int prompt_mode() {
  static const int mode = [] {
    const char* e = getenv("BSPEC_LATENT_PROMPT");
    return e != nullptr ? atoi(e) : 2;
  }();
  return mode;
}
// Decoded tokens (16- and 32-row tiles): 1 (default) = one tile of entries per CTA, so that four CTAs share an SM;
// 2 = two tiles in flight per CTA, two CTAs per SM.
static int decode_stages() {
  static const int st = [] {
    const char* e = getenv("BSPEC_LATENT_DECODE_STAGES");
    return e != nullptr && atoi(e) == 2 ? 2 : 1;
  }();
  return st;
}
BSPEC_API int bspec_latent_attention_mma_smem(int rows, int R, int P, int prompt) {
  return (int)smem_bytes(R + P, rows, (rows == 64 || (rows < 64 && !prompt && decode_stages() == 2)) ? 2 : 1);
}
static bool two_small_ctas(int R, int P) {
  return prompt_mode() == 2 && R % 32 == 0 && smem_bytes(R + P, 32, 1) <= 112 * 1024;
}

// Rows per CTA for a step whose longest portion has max_q_len tokens: 16 or 32 when every request's (token, head)
// rows fit (decoded tokens of models with few heads; needs a latent that is a multiple of 32), else 64.
BSPEC_API int bspec_latent_attention_mma_rows(int max_q_len, int H, int R, int P) {
  const long long rows = (long long)max_q_len * H;
  if (R % 32 == 0 && rows <= 16) return 16;
  if (R % 32 == 0 && rows <= 32) return 32;
  return two_small_ctas(R, P) ? 32 : 64;
}

// ``plan`` (not null: 2 ints per token of scratch, zeros where portions are left alone): the requests' keys are dealt in want_shares shares or, with more requests
// than half of that, at most one more per request; o_part and ml_part then hold (want_shares + n_entries) * max_q_len * H rows of R and of 2 floats.
// ``skip_from``: portions of that many tokens and more are left alone (``max_q_len``: the longest of the others).
BSPEC_API int bspec_latent_attention_mma(const void* ql, long long ql_row, long long ql_head, const void* qr,
                                         long long qr_row, long long qr_head, void* out, long long o_row,
                                         long long o_head, const void* cache, const int* qo_indptr,
                                         const int* positions, const int* kv_indptr, const int* kv_indices,
                                         int n_entries, int n_tokens, int max_q_len, int H, int R, int P,
                                         int page_size, float scale, float* o_part, float* ml_part,
                                         long long n_pages, const float* inv_freq, float magnitude, int window,
                                         const float* sink, int skip_from, int* plan, int want_shares,
                                         cudaStream_t stream) {
  const bool wide = prompt_mode() != 1;
  if (n_entries <= 0 || max_q_len <= 0) return 0;
  if (!bspec_latent_attention_mma_supported(R, P))
    return (int)cudaErrorInvalidValue;
  const int BM = bspec_latent_attention_mma_rows(max_q_len, H, R, P);
  const bool small_pair = BM == 32 && (long long)max_q_len * H > 32;     // prompt portions on 32-row tiles, one buffer
  const long long row_tiles = ((long long)max_q_len * H + BM - 1) / BM;
  if ((long long)max_q_len * H > 2147483647ll || n_entries > 65535) return (int)cudaErrorInvalidConfiguration;
  dim3 grid((unsigned)row_tiles, n_entries, 1);
  if (plan != nullptr) {
    if (want_shares < 1 || want_shares + n_entries > 65535 || !o_part || !ml_part) return (int)cudaErrorInvalidValue;
    grid = dim3((unsigned)row_tiles, 1, want_shares + n_entries);
  }
  const bool one_stage = small_pair || (BM < 64 && decode_stages() == 1);
  // Shares of the numbers of an entry on 16-row tiles, where as many CTAs still share an SM with the larger score tiles (a
  // decode step of 64 requests through four layers, 16 heads, latent 512 + 64: 769 -> 738 us).  With 32 rows, prompt
  // portions, the warps wait for the products rather than for their operands: 2,048 tokens 4.17 -> 4.77 ms.
  auto per_sm = [](size_t bytes) { return (int)((227 * 1024) / (bytes + 1024)); };
  const bool divide = one_stage && BM == 16 && min(4, per_sm(smem_bytes(R + P, BM, 1, 4))) >= min(4, per_sm(smem_bytes(R + P, BM, 1)));
  const size_t smem = smem_bytes(R + P, BM, one_stage ? 1 : 2, divide ? 4 : 1);
#define LM(RG, CH, N)                                                                                                \
  do {                                                                                                               \
    cudaFuncSetAttribute(latent_attn_mma_kernel<RG, CH, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    BSPEC_LAUNCH((latent_attn_mma_kernel<RG, CH, N>), grid, 32 * RG * CH, smem, stream, (const __nv_bfloat16*)ql,    \
                 ql_row, ql_head, (const __nv_bfloat16*)qr, qr_row, qr_head, (__nv_bfloat16*)out, o_row, o_head,     \
                 (const __nv_bfloat16*)cache, qo_indptr, positions, kv_indptr, kv_indices, H, R, P, page_size,       \
                 scale, o_part, ml_part, n_pages, inv_freq, magnitude, window, sink, skip_from, plan, n_entries, max_q_len * H, want_shares); \
  } while (0)
#define LMS(RG, CH, N, DS)                                                                                           \
  do {                                                                                                               \
    cudaFuncSetAttribute(latent_attn_mma_kernel<RG, CH, N, 1, DS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    BSPEC_LAUNCH((latent_attn_mma_kernel<RG, CH, N, 1, DS>), grid, 32 * RG * CH, smem, stream, (const __nv_bfloat16*)ql, \
                 ql_row, ql_head, (const __nv_bfloat16*)qr, qr_row, qr_head, (__nv_bfloat16*)out, o_row, o_head,     \
                 (const __nv_bfloat16*)cache, qo_indptr, positions, kv_indptr, kv_indices, H, R, P, page_size,       \
                 scale, o_part, ml_part, n_pages, inv_freq, magnitude, window, sink, skip_from, plan, n_entries, max_q_len * H, want_shares); \
  } while (0)
#define LM1(RG, CH, N) LMS(RG, CH, N, false)
  if (small_pair) {
    const int ntw = R / 32;
    if (ntw <= 4) LM1(2, 4, 4); else if (ntw <= 8) LM1(2, 4, 8); else LM1(2, 4, 16);
  } else if (BM == 64 && R % 32 == 0 && wide) {
    // sixteen warps: twice the warps to hide the latencies of the same tile (a warp owns a quarter of the columns)
    const int ntw = R / 32;
    if (ntw <= 4) LM(4, 4, 4); else if (ntw <= 8) LM(4, 4, 8); else LM(4, 4, 16);
  } else if (BM == 64) {
    const int ntw = R / 16;
    if (ntw <= 8) LM(4, 2, 8); else if (ntw <= 16) LM(4, 2, 16); else LM(4, 2, 32);
  } else if (one_stage) {
    const int ntw = R / 32;
    if (BM == 16 && divide) { if (ntw <= 4) LMS(1, 4, 4, true); else if (ntw <= 8) LMS(1, 4, 8, true); else LMS(1, 4, 16, true); }
    else if (BM == 16) { if (ntw <= 4) LM1(1, 4, 4); else if (ntw <= 8) LM1(1, 4, 8); else LM1(1, 4, 16); }
    else { if (ntw <= 4) LM1(2, 4, 4); else if (ntw <= 8) LM1(2, 4, 8); else LM1(2, 4, 16); }
  } else {
    const int ntw = R / 32;
    if (BM == 16) { if (ntw <= 4) LM(1, 4, 4); else if (ntw <= 8) LM(1, 4, 8); else LM(1, 4, 16); }
    else { if (ntw <= 4) LM(2, 4, 4); else if (ntw <= 8) LM(2, 4, 8); else LM(2, 4, 16); }
  }
#undef LM1
#undef LMS
#undef LM
  int err = BSPEC_LAUNCH_CHECK();
  if (err != 0 || plan == nullptr) return err;
  const long long rows = (long long)n_tokens * H, fit = 16ll * bspec::sm_count();
  if (rows > 2147483647ll) return (int)cudaErrorInvalidConfiguration;
  const int per_block = rows <= fit ? 1 : 4;
  BSPEC_LAUNCH((latent_attn_join_kernel), (unsigned)min((rows + per_block - 1) / per_block, fit), 128, 0, stream, o_part, ml_part,
               (__nv_bfloat16*)out, o_row, o_head, H, R, (const int*)plan, max_q_len * H, (int)rows, per_block);
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_DEFINE_TRACE_SETTER(bspec_trace_set_latent_mma)
BSPEC_DEFINE_BOUNDS_REPORT(bspec_bounds_report_latent_mma)
