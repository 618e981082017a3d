// Recurrences with one matrix of state per head, S [key rows x value columns] float32, taken tile by tile: what eight tokens
// read from S is formed before any of them writes, and their effect on one another comes in through small matrices that
// are the same for every value column (the caller's preparation kernel forms them once per tile and head).  Per tile, with
// a_t = S^T k_t (where the rule reads it; RK) and b_t = S^T q_t,
//     x_t = e_t v_t - d_t a_t,     o_t = c_t b_t + sum_s P_ts x_s,     S <- c_B S + sum_t k_t w_t^T,  w_t = sum_s F_ts x_s.
#pragma once
#include "common.cuh"
#include <cuda_pipeline.h>

namespace bspec {

// tokens of a tile; floats of a token's row of coefficients [F_t 8 | P_t 8 | d_t, e_t, c_t, c_B]; floats of a tile's
constexpr int ST_B = 8, ST_ROW = 20, ST_CO = ST_B * ST_ROW;
// In a step whose long portions go by tiles (tiles_pay) those are the portions of at least ST_FROM tokens.
constexpr int ST_FROM = 64;
constexpr int ST_COLS = 16, ST_STAGE = 16, ST_THREADS = 128;

// Where tile i of entry e has its coefficients (times heads): tiles of different entries never meet.
__device__ __forceinline__ size_t state_tile_slot(int q_begin, int e, int i) { return (size_t)(q_begin / ST_B + e + i); }
inline long long state_tile_slots(int n, int n_entries) { return n / ST_B + n_entries + 1; }

// The entry whose slots hold ``slot``: the last one that begins at or before it.  (The preparation kernels' grids go over the
// slots: over the tiles of the longest portion times the requests, a portion of 8,192 tokens beside 63 decoded ones was a
// million blocks with 16,384 tiles to form.)  A warp looks at 32 entries at a time.
__device__ __forceinline__ int state_tile_entry(const int* __restrict__ qo_indptr, int n_entries, int slot) {
  const int lane = threadIdx.x & 31;
  int first = 0, count = n_entries;                            // the answer is one of ``count`` entries from ``first`` on
  while (count > 1) {
    const int step = (count + 31) / 32, e = first + lane * step;
    const unsigned before = __ballot_sync(0xffffffffu, lane * step < count && (int)state_tile_slot(qo_indptr[min(e, n_entries - 1)], e, 0) <= slot);
    const int k = max(0, 31 - __clz(before));
    first += k * step;
    count = min(step, count - k * step);
  }
  return first;
}

// What a token takes, us on a B200: ``chain`` in a portion's chain, ``rate`` times heads x rows of the instance x value columns when
// the device is full.
struct TokenCost {
  double chain, rate;
};

struct Tall {                    // the most portions of ST_FROM tokens and more, the tokens in them, what the others than the longest have beyond ``least`` each
  long long count;
  double tokens;
  long long rest;
  int least;
};
inline Tall tall_portions(int n, int n_entries, int shortest, int longest) {
  Tall t;
  t.least = shortest < 1 ? 1 : shortest;
  const long long spare = (long long)n - longest - (long long)(n_entries - 1) * t.least;
  t.rest = spare < 0 ? 0 : spare;
  t.count = 1;
  if (t.least >= ST_FROM) t.count = n_entries;
  else t.count += t.rest / (ST_FROM - t.least) < n_entries - 1 ? t.rest / (ST_FROM - t.least) : n_entries - 1;
  t.tokens = (double)n - (double)(n_entries - t.count) * t.least;
  return t;
}

// Whether a step is faster with its long portions by tiles.  Tiles have the shorter chain, 8 tokens in about a microsecond, but
// one instance for all heads of up to 128 rows, a preparation, and a second kernel for the shorter portions; token loops have
// instances for 32 and 64 rows.  So both are estimated, as the longer of a chain and the work of a full device.  The constants are
// fitted to 594 measured steps (1 to 64 heads of 32 to 256, 1 to 64 requests of 1 to 8,192 tokens); where the choice is wrong the
// other form is less than 5 us or a sixth faster.  By tokens / by tiles, us, delta rule and lightning attention:
//   16 heads of 128 x 128: 1 x 64 19 / 14 and 18 / 15; 2,048 beside 24 decoded 666 / 388 and 853 / 358; 32 x 128 344 / 314 and 485 / 306
//   16 heads of 64 x 64: 1 x 64 13 / 14; 32 x 64 53 / 90 and 61 / 88; 4 x 2,048 577 / 412 and 550 / 389
//   64 heads of 64 x 64: 32 x 128 374 / 660 and 448 / 618; 2,048 beside 63 653 / 548 and 628 / 513; 128 beside 63 (lightning) 47 / 76
//   32 heads of 32 x 32 (lightning): 32 x 64 40 / 97; 512 beside 63 88 / 76
//   8 heads of 256 x 256: 32 x 64 354 / 315 and 733 / 262; 64 tokens beside twenty of 60, any heads: a loss, 119 / 137 at 16 x 128
// (A step is what the estimate needs; a request's results differ by rounding between the two forms.)
inline bool tiles_pay(int n, int n_entries, int shortest, int longest, int H, int dim, int vdim, TokenCost tokens, TokenCost tiles) {
  if (longest < ST_FROM) return false;
  const Tall t = tall_portions(n, n_entries, shortest, longest);
  const int least = t.least;
  const long long rest = t.rest;
  const double tiled = t.tokens;
  const int rows = dim <= 32 ? 32 : (dim <= 64 ? 64 : (dim <= 128 ? 128 : 256));
  const double token_work = (double)H * rows * vdim * tokens.rate, tile_work = (double)H * ((vdim + 15) / 16) * tiles.rate;
  auto longer = [](double a, double b) { return a > b ? a : b; };
  const double by_tokens = longer(longest * tokens.chain, n * token_work) + 4.0;
  double by_tiles = longer(longest * tiles.chain, tiled * tile_work) + tiled * H * (0.5e-4 + 2e-6 * dim) + 7.5;
  if (least < ST_FROM && n_entries > 1) {                                                   // the second kernel
    const double s = least + rest < ST_FROM - 1 ? (double)(least + rest) : ST_FROM - 1;
    by_tiles += 3.0 + longer(s * tokens.chain, (n - tiled) * token_work) + (double)(n_entries - 1) * H * dim * vdim / 3e6;
  }
  return by_tiles < by_tokens;
}

constexpr size_t state_tiles_smem(int dp) {
  return (size_t)(2 * ST_STAGE * (2 * dp + ST_COLS) + 2 * (ST_STAGE / ST_B) * ST_CO + 4 * 64 * 16 + 4 * 32) * 4;
}

struct StateTiles {
  const float *q, *k, *v;              // this head's first number of the portion's first token
  long long q_stride, k_stride, v_stride;
  const float* coef;                   // the portion's first tile
  long long coef_stride;
  float* s;                            // column 0 of this head's S
  int s_stride, s_rows;                // a column's numbers in memory (rows from dim to s_rows are zeros)
  float* out;                          // column 0 of this head, the portion's first token
  long long out_stride;
  int n, dim, vdim, j0;                // tokens; sizes of the head; first value column of the block
};

// Block of four warps, four value columns per warp: half warp g holds columns 2 g and 2 g + 1, its lane r rows
// 64 c + 4 r + {0..3} of both, R of them.  Per tile a lane forms its share of the sums a and b (2 columns x 8 tokens each) and
// leaves them in shared memory; then lane 8 x + t adds up the a and b of one column and token t over the half warp's lanes,
// gets the tile's x from its neighbours and forms o and w.  Bound by shared memory and by the chain of a tile: 16
// lanes per column instead of 32 halve both the sums' way through shared memory and the reads of q and k per column.
// The sums lie in rows of 16 floats without padding: the half warps write to different halves of the banks (row t ^ g), the
// quads of a row are turned by the row's number, so that neither the writes nor the 16-byte reads collide.  Tokens are
// staged 16 at a time, the next stage under the current one.  2,048 tokens of 16 heads of 128 x 128 on a B200, with the
// preparation: 261 us (delta rule; 435 us beside requests of 333 and 826 tokens, 753 us token by token) and 263 us (lightning
// attention; 553 us).  Eight warps of two columns each took as long alone and a tenth more beside the two.
template <int R, bool RK, typename Act>
__device__ __forceinline__ void state_tiles(const StateTiles& p, Act act) {
  constexpr int NT = ST_THREADS, DP = 16 * R;
  constexpr bool HOLD = R <= 8;                                // the tile's keys stay in registers for the update
  extern __shared__ __align__(16) float smem_f[];
  float* qs = smem_f;                                          // [2][STAGE][DP]
  float* ks = qs + 2 * ST_STAGE * DP;                          // [2][STAGE][DP]
  float* vs = ks + 2 * ST_STAGE * DP;                          // [2][STAGE][COLS]
  float* cs = vs + 2 * ST_STAGE * ST_COLS;                     // [2][STAGE / B][CO]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* sums = cs + 2 * (ST_STAGE / ST_B) * ST_CO + warp * 64 * 16;                     // [a, b][2][8 g + token ^ g][16] of this warp
  float* wb = cs + 2 * (ST_STAGE / ST_B) * ST_CO + 4 * 64 * 16 + warp * 32;              // [4 columns][8 tokens] of this warp
  const int n = p.n, dim = p.dim, g = lane >> 4, r16 = lane & 15;
  for (int w = tid; w < 2 * ST_STAGE * (DP - dim); w += NT) {  // the pad of a row is never copied into
    const int bt = w / (DP - dim), d = dim + w % (DP - dim);
    qs[bt * DP + d] = 0.f;
    ks[bt * DP + d] = 0.f;
  }
  // rows of q and k start on 16-byte boundaries
  const bool vec = ((dim | (int)p.q_stride | (int)p.k_stride) & 3) == 0 && (((uintptr_t)p.q | (uintptr_t)p.k) & 15) == 0;
  // this thread's first copies of a whole stage: token warp of q and k, token tid / 16 of v, a quad of the coefficients
  const float *q_src = p.q + warp * p.q_stride + 4 * lane, *k_src = p.k + warp * p.k_stride + 4 * lane;
  const int v_tok = tid / ST_COLS, v_col = p.j0 + tid % ST_COLS;
  const float* v_src = p.v + v_tok * p.v_stride + v_col;
  const int c_half = tid / (ST_CO / 4), c_off = tid % (ST_CO / 4) * 4;
  auto stage = [&](int t0, int buf) {                          // tokens t0 .. t0 + STAGE - 1 of the portion, zeros past its end
    const int nt = min(ST_STAGE, n - t0);
    if (vec && nt == ST_STAGE) {                               // (the general form below took a sixth of the kernel's time)
      const float *qr = q_src + t0 * p.q_stride, *kr = k_src + t0 * p.k_stride, *vr = v_src + t0 * p.v_stride;
      float *qd = qs + (buf * ST_STAGE + warp) * DP + 4 * lane, *kd = ks + (buf * ST_STAGE + warp) * DP + 4 * lane;
#pragma unroll
      for (int i = 0; i < ST_STAGE / (NT / 32); ++i)
#pragma unroll
        for (int d = 0; d < DP; d += 128)
          if (d + 4 * lane < dim) {
            __pipeline_memcpy_async(qd + i * (NT / 32) * DP + d, qr + i * (NT / 32) * p.q_stride + d, 16);
            __pipeline_memcpy_async(kd + i * (NT / 32) * DP + d, kr + i * (NT / 32) * p.k_stride + d, 16);
          }
#pragma unroll
      for (int i = 0; i < ST_STAGE * ST_COLS / NT; ++i) {
        float* vd = vs + buf * ST_STAGE * ST_COLS + tid + i * NT;
        if (v_col < p.vdim) __pipeline_memcpy_async(vd, vr + i * (NT / ST_COLS) * p.v_stride, 4);
        else *vd = 0.f;
      }
      if (c_half < ST_STAGE / ST_B)
        __pipeline_memcpy_async(cs + (buf * (ST_STAGE / ST_B) + c_half) * ST_CO + c_off, p.coef + (t0 / ST_B + c_half) * p.coef_stride + c_off, 16);
      __pipeline_commit();
      return;
    }
    for (int tt = warp; tt < ST_STAGE; tt += NT / 32) {
      const float *qr = p.q + (t0 + min(tt, nt - 1)) * p.q_stride, *kr = p.k + (t0 + min(tt, nt - 1)) * p.k_stride;
      float *qd = qs + (buf * ST_STAGE + tt) * DP, *kd = ks + (buf * ST_STAGE + tt) * DP;
      if (tt >= nt) {
        for (int d = lane; d < dim; d += 32) qd[d] = kd[d] = 0.f;
      } else if (vec) {
        for (int d = 4 * lane; d < dim; d += 128) {
          __pipeline_memcpy_async(qd + d, qr + d, 16);
          __pipeline_memcpy_async(kd + d, kr + d, 16);
        }
      } else {
        for (int d = lane; d < dim; d += 32) {
          __pipeline_memcpy_async(qd + d, qr + d, 4);
          __pipeline_memcpy_async(kd + d, kr + d, 4);
        }
      }
    }
    for (int w = tid; w < ST_STAGE * ST_COLS; w += NT) {
      const int tt = w / ST_COLS, jj = p.j0 + w % ST_COLS;
      float* vd = vs + buf * ST_STAGE * ST_COLS + w;
      if (tt < nt && jj < p.vdim) __pipeline_memcpy_async(vd, p.v + (t0 + tt) * p.v_stride + jj, 4);
      else *vd = 0.f;
    }
    for (int w = tid; w < (ST_STAGE / ST_B) * (ST_CO / 4); w += NT) {
      const int half = w / (ST_CO / 4), x = w % (ST_CO / 4) * 4;
      if (half * ST_B < nt)
        __pipeline_memcpy_async(cs + (buf * (ST_STAGE / ST_B) + half) * ST_CO + x, p.coef + (t0 / ST_B + half) * p.coef_stride + x, 16);
    }
    __pipeline_commit();
  };
  stage(0, 0);
  const bool svec = (p.s_stride & 3) == 0 && ((uintptr_t)p.s & 15) == 0;
  float s[2][R];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int j = p.j0 + 4 * warp + 2 * g + c;
    const float* sp = p.s + (size_t)(j < p.vdim ? j : 0) * p.s_stride;
#pragma unroll
    for (int q = 0; q < R / 4; ++q) {
      const int row = 64 * q + 4 * r16;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < p.vdim && row < p.s_rows) {
        if (svec) v = *reinterpret_cast<const float4*>(sp + row);
        else v = make_float4(sp[row], row + 1 < p.s_rows ? sp[row + 1] : 0.f, row + 2 < p.s_rows ? sp[row + 2] : 0.f,
                             row + 3 < p.s_rows ? sp[row + 3] : 0.f);
      }
      s[c][4 * q] = v.x, s[c][4 * q + 1] = v.y, s[c][4 * q + 2] = v.z, s[c][4 * q + 3] = v.w;
    }
  }
  // what this lane finishes: column lane / 8 of the warp (half warp (lane / 8) % 2, its column lane / 16), token lane % 8
  const int tok = lane & 7, own = 2 * ((lane >> 3) & 1) + (lane >> 4), j = p.j0 + 4 * warp + own;
  const int own_row = (lane >> 4) * 16 + ((lane >> 3) & 1) * 8 + (tok ^ ((lane >> 3) & 1)), own_turn = (own_row >> 1) & 3;
  int buf = 0;
  for (int t0 = 0; t0 < n; t0 += ST_STAGE, buf ^= 1) {
    __pipeline_wait_prior(0);
    __syncthreads();                                           // the stage is there, and every thread is done with the other half
    if (t0 + ST_STAGE < n) stage(t0 + ST_STAGE, buf ^ 1);
#pragma unroll
    for (int half = 0; half < ST_STAGE / ST_B && t0 + half * ST_B < n; ++half) {
      const float* kt = ks + (buf * ST_STAGE + half * ST_B) * DP + 4 * r16;
      const float* qt = qs + (buf * ST_STAGE + half * ST_B) * DP + 4 * r16;
      float k[HOLD ? ST_B : 1][R];
#pragma unroll
      for (int t = 0; t < ST_B; ++t) {
        float q[R];
        float (&kk)[R] = k[HOLD ? t : 0];
#pragma unroll
        for (int x = 0; x < R / 4; ++x) {
          const float4 k4 = *reinterpret_cast<const float4*>(kt + t * DP + 64 * x);
          const float4 q4 = *reinterpret_cast<const float4*>(qt + t * DP + 64 * x);
          kk[4 * x] = k4.x, kk[4 * x + 1] = k4.y, kk[4 * x + 2] = k4.z, kk[4 * x + 3] = k4.w;
          q[4 * x] = q4.x, q[4 * x + 1] = q4.y, q[4 * x + 2] = q4.z, q[4 * x + 3] = q4.w;
        }
        // row 8 g + (t ^ g) of 16 floats, its quads turned by the row's number
        float* at = sums + (8 * g + (t ^ g)) * 16 + (((r16 >> 2) ^ ((t >> 1) & 3)) << 2) + (r16 & 3);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float a = 0.f, b = s[c][0] * q[0];
          if (RK) a = s[c][0] * kk[0];
#pragma unroll
          for (int r = 1; r < R; ++r) {
            if (RK) a = fmaf(s[c][r], kk[r], a);
            b = fmaf(s[c][r], q[r], b);
          }
          if (RK) at[c * 256] = a;
          at[512 + c * 256] = b;
        }
      }
      const float* co = cs + (buf * (ST_STAGE / ST_B) + half) * ST_CO + tok * ST_ROW;
      float f[2 * ST_B];                                       // the token's rows of F and of P
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float4 v = *reinterpret_cast<const float4*>(co + 4 * x);
        f[4 * x] = v.x, f[4 * x + 1] = v.y, f[4 * x + 2] = v.z, f[4 * x + 3] = v.w;
      }
      const float4 cc = *reinterpret_cast<const float4*>(co + 16);             // d_t, e_t, c_t, c_B
      const float vj = act(vs[(buf * ST_STAGE + half * ST_B + tok) * ST_COLS + 4 * warp + own]);
      __syncwarp();
      float4 a4 = make_float4(0.f, 0.f, 0.f, 0.f), b4 = a4;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float4 v = *reinterpret_cast<const float4*>(sums + 512 + own_row * 16 + ((x ^ own_turn) << 2));
        b4.x += v.x, b4.y += v.y, b4.z += v.z, b4.w += v.w;
        if (RK) {
          const float4 u = *reinterpret_cast<const float4*>(sums + own_row * 16 + ((x ^ own_turn) << 2));
          a4.x += u.x, a4.y += u.y, a4.z += u.z, a4.w += u.w;
        }
      }
      float x = cc.y * vj;
      if (RK) x -= cc.x * ((a4.x + a4.y) + (a4.z + a4.w));
      float w = 0.f, o = cc.z * ((b4.x + b4.y) + (b4.z + b4.w));
#pragma unroll
      for (int t = 0; t < ST_B; ++t) {
        const float xs = __shfl_sync(0xffffffffu, x, (lane & 24) | t);
        const float xt = t <= tok ? xs : 0.f;                  // (a later token's x may be anything)
        w = fmaf(f[t], xt, w);
        o = fmaf(f[ST_B + t], xt, o);
      }
      wb[own * ST_B + tok] = w;
      if (t0 + half * ST_B + tok < n && j < p.vdim) p.out[(t0 + half * ST_B + tok) * p.out_stride + j] = o;
      __syncwarp();
      float wt[2][ST_B];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float4 w0 = *reinterpret_cast<const float4*>(wb + (2 * g + c) * ST_B);
        const float4 w1 = *reinterpret_cast<const float4*>(wb + (2 * g + c) * ST_B + 4);
        wt[c][0] = w0.x, wt[c][1] = w0.y, wt[c][2] = w0.z, wt[c][3] = w0.w;
        wt[c][4] = w1.x, wt[c][5] = w1.y, wt[c][6] = w1.z, wt[c][7] = w1.w;
#pragma unroll
        for (int r = 0; r < R; ++r) s[c][r] *= cc.w;
      }
#pragma unroll
      for (int t = 0; t < ST_B; ++t) {
        if (!HOLD) {
#pragma unroll
          for (int y = 0; y < R / 4; ++y) {
            const float4 k4 = *reinterpret_cast<const float4*>(kt + t * DP + 64 * y);
            k[0][4 * y] = k4.x, k[0][4 * y + 1] = k4.y, k[0][4 * y + 2] = k4.z, k[0][4 * y + 3] = k4.w;
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int r = 0; r < R; ++r) s[c][r] = fmaf(k[HOLD ? t : 0][r], wt[c][t], s[c][r]);
      }
    }
  }
  pdl_launch_dependents();
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int jc = p.j0 + 4 * warp + 2 * g + c;
    float* sp = p.s + (size_t)jc * p.s_stride;
#pragma unroll
    for (int q = 0; q < R / 4; ++q) {
      const int row = 64 * q + 4 * r16;
      if (jc < p.vdim && row < p.s_rows) {
        if (svec) {
          *reinterpret_cast<float4*>(sp + row) = make_float4(s[c][4 * q], s[c][4 * q + 1], s[c][4 * q + 2], s[c][4 * q + 3]);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (row + u < p.s_rows) sp[row + u] = s[c][4 * q + u];
        }
      }
    }
  }
}

}  // namespace bspec
