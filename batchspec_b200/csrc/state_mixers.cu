// Two recurrent mixers whose state per request has a fixed size, float32 throughout.
//
//   lightning_recurrence   linear attention with a fixed decay per head:
//                              S <- decay_h S + k v^T,  o = S^T q        S: [dim x vdim] per head
//                          q, k, v are float32 projection columns, through silu or as they are; q and k may be
//                          rotated by position (pairs i, i + rot/2) and k multiplied by a constant.
//   scan_conv              short causal convolution per channel with bias, then silu (inputs before the portion come
//                          from the request's state)
//   selective_scan         per channel c and state n:  S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n,
//                              y_c = sum_n S[c, n] C_n + D_c x_c,  out_c = y_c silu(z_c),  dt = softplus(raw + bias),
//                              A = -exp(A_log)
//
// A step holds portions of several requests (qo_indptr, state_slots); a portion of one token is a decode step.
// Which form runs depends on the portion's length and, through the estimates of their times, on the step's tokens, its requests
// and the sizes: lightning attention token by token, by tiles or by chunks, the scan end to end or in segments, lanes per column or
// channel.  Within a form the order of every sum is fixed; between forms, so between ways to cut a request into portions and
// between neighbours in a step, results differ by float32 rounding.
#include "state_chunks.cuh"
#include <math.h>
using namespace bspec;

namespace {

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
// S <- exp(x) S + b as S + ((exp(x) - 1) S + b).  A state with a long memory has exp(x) within 1e-4 of 1, where a
// float32 factor keeps only three digits of what matters, 1 - exp(x); taken a thousand times that shows in the sum.
// exp(x) - 1 keeps all its digits, and the state moves by the small difference.
// Near zero exp(x) - 1 is the series up to x^4 / 24 (the next term is below 1e-8 of the sum for |x| < 1/32); further
// out 2^(x log2 e) - 1, whose difference from 1 is large enough to keep its digits.
__device__ __forceinline__ float exp_minus_one(float x) {
  const float series = __fmul_rn(x, __fmaf_rn(x, __fmaf_rn(x, __fmaf_rn(x, 1.f / 24.f, 1.f / 6.f), 0.5f), 1.f));
  const float direct = exp2f(__fmul_rn(x, 1.4426950408889634f)) - 1.f;
  return fabsf(x) < 0.03125f ? series : direct;
}
__device__ __forceinline__ float scan_update(float s, float x, float b) {
  return __fadd_rn(s, __fmaf_rn(exp_minus_one(x), s, b));
}

// The angle position * frequency in float64 (the table holds a frequency as two float32 parts), reduced to [-pi, pi].
__device__ __forceinline__ void rotation_sincos(int pos, const float* __restrict__ inv_freq, int half, int j, float* s,
                                                float* c) {
  const double f = (double)inv_freq[j] + (double)inv_freq[half + j];
  double a = (double)pos * f;
  a -= 6.283185307179586476925286766559 * rint(a * 0.15915494309189533576888376337251);
  sincosf((float)a, s, c);
}

// ---------------------------------------------------------------- lightning attention
// Block: COLS value columns of one head of one request, L lanes per column (8, 16 or 32: more lanes mean more warps
// per SM to hide the chain's latencies, and fewer rows per lane); lane r of a column keeps rows
// 4 L g + 4 r + e (e < 4, g < NR / 4) of that column of S in registers, so that a lane reads its four rows of q and k
// from shared memory in one 16-byte load.  Tokens are staged TT at a time in shared memory: the raw projection
// columns of the next TT tokens are fetched into registers while the recurrence runs over the current ones, so the
// memory latency is paid once per kernel and not once per batch of tokens.  The recurrence takes four tokens per
// pass (sixteen independent chains of four dependent multiply-adds); a token's sums run in the same order in the
// four-token pass and in the single-token tail, so a position's result does not depend on where a portion ends.
// State of a request: [H][vdim][dim] float32 at state + slot * state_stride.
constexpr int LT_COLS = 16;
constexpr int LT_TT = 16;

template <int NR, int L>
__global__ void __launch_bounds__(LT_COLS * L)
lightning_recurrence_kernel(const float* __restrict__ proj, long long ld, int q_off, int k_off, int v_off,
                            const float* __restrict__ decay, float* __restrict__ state, long long state_stride,
                            const int* __restrict__ qo_indptr, const int* __restrict__ state_slots,
                            float* __restrict__ out, int H, int dim, int vdim, int act, float k_scale,
                            const float* __restrict__ inv_freq, int rot, const int* __restrict__ positions, int below) {
  bspec::pdl_prologue_late(65);
  constexpr int LT_THREADS = LT_COLS * L;
  constexpr int DM = L * NR;                                // rows of S this instance holds (dim <= DM)
  constexpr int VR = (LT_TT * LT_COLS + LT_THREADS - 1) / LT_THREADS;          // staged v values per thread
  static_assert(NR % 4 == 0 && (L == 8 || L == 16 || L == 32) && LT_TT * DM == NR * LT_THREADS, "lanes and rows");
  __shared__ __align__(16) float qs[LT_TT][DM];
  __shared__ __align__(16) float ks[LT_TT][DM];
  __shared__ float vs[LT_TT][LT_COLS];
  const int e = blockIdx.z, h = blockIdx.y;
  const int col = threadIdx.x / L, r = threadIdx.x % L;
  const int j = blockIdx.x * LT_COLS + col;                 // value column of the head
  const bool live = j < vdim;
  const int t0 = qo_indptr[e], nt = qo_indptr[e + 1] - t0;
  if (nt >= below) return;                                  // the portion goes by tiles
  const float d = decay[h];
  float* sp = state + (size_t)state_slots[e] * state_stride + ((size_t)h * vdim + (live ? j : 0)) * dim;
  float qn[NR], kn[NR], vn[VR];
  // the raw columns of tokens base .. base + TT - 1 (zeros beyond the portion, the head's rows and the columns)
  auto fetch = [&](int base) {
    const int cnt = min(LT_TT, nt - base);
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const int x = threadIdx.x + LT_THREADS * u;
      const int tt = x / DM, i = x % DM;                     // tt is the same for a whole warp (DM >= 32)
      if (tt >= cnt) break;
      const bool ok = i < dim;
      const float* row = proj + (size_t)(t0 + base + tt) * ld + (size_t)h * dim + (ok ? i : 0);
      qn[u] = ok ? row[q_off] : 0.f;
      kn[u] = ok ? row[k_off] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < VR; ++u) {
      const int x = threadIdx.x + LT_THREADS * u;
      const int tt = x / LT_COLS, c = x % LT_COLS;
      const int jj = blockIdx.x * LT_COLS + c;
      const bool ok = x < LT_TT * LT_COLS && tt < cnt && jj < vdim;
      vn[u] = ok ? proj[(size_t)(t0 + base + tt) * ld + v_off + (size_t)h * vdim + jj] : 0.f;
    }
  };
  if (nt > 0) fetch(0);
  float s[NR];
  const bool vec = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(sp) & 15) == 0;
  if (vec) {
#pragma unroll
    for (int g = 0; g < NR / 4; ++g) {
      const int i = 4 * L * g + 4 * r;
      const float4 v4 = (live && i < dim) ? *reinterpret_cast<const float4*>(sp + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      s[4 * g] = v4.x, s[4 * g + 1] = v4.y, s[4 * g + 2] = v4.z, s[4 * g + 3] = v4.w;
    }
  } else {
#pragma unroll
    for (int m = 0; m < NR; ++m) {
      const int i = 4 * L * (m >> 2) + 4 * r + (m & 3);
      s[m] = (live && i < dim) ? sp[i] : 0.f;
    }
  }
  for (int base = 0; base < nt; base += LT_TT) {
    const int cnt = min(LT_TT, nt - base);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < NR; ++u) {                           // rows of tokens beyond cnt are never read
      const int x = threadIdx.x + LT_THREADS * u;
      if (x / DM >= cnt) break;
      qs[x / DM][x % DM] = act ? silu_f(qn[u]) : qn[u];      // silu(0) = 0: rows beyond dim
      ks[x / DM][x % DM] = (act ? silu_f(kn[u]) : kn[u]) * k_scale;
    }
#pragma unroll
    for (int u = 0; u < VR; ++u) {
      const int x = threadIdx.x + LT_THREADS * u;
      if (x < LT_TT * LT_COLS && x / LT_COLS < cnt) vs[x / LT_COLS][x % LT_COLS] = act ? silu_f(vn[u]) : vn[u];
    }
    __syncthreads();
    if (rot > 0) {                                           // the same for every block of a head: meant for a few tokens
      const int half = rot / 2;
      for (int x = threadIdx.x; x < cnt * half; x += LT_THREADS) {
        const int tt = x / half, i = x - tt * half;
        float sn, c;
        rotation_sincos(positions[t0 + base + tt], inv_freq, half, i, &sn, &c);
        const float qu = qs[tt][i], qv = qs[tt][i + half], ku = ks[tt][i], kv = ks[tt][i + half];
        qs[tt][i] = qu * c - qv * sn;
        qs[tt][i + half] = qv * c + qu * sn;
        ks[tt][i] = ku * c - kv * sn;
        ks[tt][i + half] = kv * c + ku * sn;
      }
      __syncthreads();
    }
    if (base + LT_TT < nt) fetch(base + LT_TT);
    float* orow = out + (size_t)(t0 + base) * H * vdim + (size_t)h * vdim + j;
    int tt = 0;
    for (; tt + 4 <= cnt; tt += 4) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f}, vj[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) vj[a] = vs[tt + a][col];
#pragma unroll
      for (int g = 0; g < NR / 4; ++g) {
        float4 k4[4], q4[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          k4[a] = *reinterpret_cast<const float4*>(&ks[tt + a][4 * L * g + 4 * r]);
          q4[a] = *reinterpret_cast<const float4*>(&qs[tt + a][4 * L * g + 4 * r]);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const float kk[4] = {k4[a].x, k4[a].y, k4[a].z, k4[a].w}, qq[4] = {q4[a].x, q4[a].y, q4[a].z, q4[a].w};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            s[4 * g + c] = __fmaf_rn(d, s[4 * g + c], __fmul_rn(kk[c], vj[a]));
            acc[a] = __fmaf_rn(s[4 * g + c], qq[c], acc[a]);
          }
        }
      }
#pragma unroll
      for (int o = 1; o < L; o <<= 1)
#pragma unroll
        for (int a = 0; a < 4; ++a) acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], o);
      const float mine = r == 0 ? acc[0] : (r == 1 ? acc[1] : (r == 2 ? acc[2] : acc[3]));
      if (live && r < 4) orow[(size_t)(tt + r) * H * vdim] = mine;
    }
    for (; tt < cnt; ++tt) {
      const float vj = vs[tt][col];
      float acc = 0.f;
#pragma unroll
      for (int g = 0; g < NR / 4; ++g) {
        const float4 k4 = *reinterpret_cast<const float4*>(&ks[tt][4 * L * g + 4 * r]);
        const float4 q4 = *reinterpret_cast<const float4*>(&qs[tt][4 * L * g + 4 * r]);
        const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, qq[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          s[4 * g + c] = __fmaf_rn(d, s[4 * g + c], __fmul_rn(kk[c], vj));
          acc = __fmaf_rn(s[4 * g + c], qq[c], acc);
        }
      }
#pragma unroll
      for (int o = 1; o < L; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (live && r == 0) orow[(size_t)tt * H * vdim] = acc;
    }
  }
  bspec::pdl_launch_dependents();
  if (live && vec) {
#pragma unroll
    for (int g = 0; g < NR / 4; ++g) {
      const int i = 4 * L * g + 4 * r;
      if (i < dim) *reinterpret_cast<float4*>(sp + i) = make_float4(s[4 * g], s[4 * g + 1], s[4 * g + 2], s[4 * g + 3]);
    }
  } else if (live) {
#pragma unroll
    for (int m = 0; m < NR; ++m) {
      const int i = 4 * L * (m >> 2) + 4 * r + (m & 3);
      if (i < dim) sp[i] = s[m];
    }
  }
}

// ---------------------------------------------------------------- lightning attention, portions of whole tiles
// The token loop above is bound by its four-token passes' shared-memory loads and latencies (270 ns a token: 553 us for 2,048
// tokens, 16 heads of 128 x 128).  Eight tokens at a time (state_tiles.cuh): x = v, F = diag(d^(B-1-t)), P_ts = d^(t-s)
// (k_s . q_t), c_t = d^(t+1).  A tile of ``cnt`` < 8 tokens counts the others as zeros without decay.  The preparation
// kernel, one block per (tile, head), also leaves q and k as the recurrence wants them (silu, scale, rotation), which every
// block of a head would repeat otherwise: qk [n][H][q: dim | k: dim].
__global__ void __launch_bounds__(128)
lightning_tiles_prepare_kernel(const float* __restrict__ proj, long long ld, int q_off, int k_off, const float* __restrict__ decay,
                               const int* __restrict__ qo_indptr, int n_entries, float* __restrict__ qk, float* __restrict__ coef,
                               int H, int dim, int act, float k_scale, const float* __restrict__ inv_freq, int rot, const int* __restrict__ positions) {
  bspec::pdl_prologue(65);
  __shared__ float qs[ST_B][264], ks[ST_B][264], dots[ST_B][ST_B];      // (rows eight banks apart)
  const int h = blockIdx.y, e = state_tile_entry(qo_indptr, n_entries, blockIdx.x);
  const int q_begin = qo_indptr[e], n = qo_indptr[e + 1] - q_begin, i = blockIdx.x - (int)state_tile_slot(q_begin, e, 0);
  if (n < ST_FROM || i * ST_B >= n) return;                    // (i >= 0: the first entry's slots begin at 0)
  const int cnt = min(ST_B, n - i * ST_B), t0 = q_begin + i * ST_B;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int u = 0; u < ST_B / 4; ++u) {
    const int t = warp + 4 * u;
    const float* row = proj + (size_t)(t0 + min(t, cnt - 1)) * ld + (size_t)h * dim;
    for (int d = lane; d < dim; d += 32) {
      const float q = row[q_off + d], k = row[k_off + d];
      qs[t][d] = t < cnt ? (act ? silu_f(q) : q) : 0.f;
      ks[t][d] = t < cnt ? (act ? silu_f(k) : k) * k_scale : 0.f;
    }
  }
  __syncthreads();
  if (rot > 0) {
    const int half = rot / 2;
    for (int x = tid; x < cnt * half; x += 128) {
      const int t = x / half, d = x - t * half;
      float sn, c;
      rotation_sincos(positions[t0 + t], inv_freq, half, d, &sn, &c);
      const float qu = qs[t][d], qv = qs[t][d + half], ku = ks[t][d], kv = ks[t][d + half];
      qs[t][d] = qu * c - qv * sn;
      qs[t][d + half] = qv * c + qu * sn;
      ks[t][d] = ku * c - kv * sn;
      ks[t][d + half] = kv * c + ku * sn;
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < ST_B / 4; ++u) {
    const int t = warp + 4 * u;
    float* row = qk + ((size_t)(t0 + t) * H + h) * 2 * dim;
    for (int d = lane; t < cnt && d < dim; d += 32) {
      row[d] = qs[t][d];
      row[dim + d] = ks[t][d];
    }
  }
  // a warp takes two t, eight lanes a dot (four s at a time)
#pragma unroll
  for (int u = 0; u < ST_B / 2; ++u) {
    const int t = 2 * warp + u / 2, s = 4 * (u & 1) + lane / 8;
    float a = 0.f;
    for (int d = lane % 8; d < dim; d += 8) a = fmaf(ks[s][d], qs[t][d], a);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane % 8 == 0) dots[t][s] = a;
  }
  __syncthreads();
  float* co = coef + (state_tile_slot(q_begin, e, i) * H + h) * ST_CO;
  if (tid < ST_B * ST_B) {
    const int t = tid / ST_B, s = tid % ST_B;
    const float d = decay[h];
    float pw[ST_B + 1];                                        // d^0 .. d^8
    pw[0] = 1.f;
#pragma unroll
    for (int u = 0; u < ST_B; ++u) pw[u + 1] = pw[u] * d;
    auto power = [&](int u) {
      float v = 1.f;
#pragma unroll
      for (int x = 1; x <= ST_B; ++x) v = u == x ? pw[x] : v;
      return v;
    };
    co[t * ST_ROW + s] = s == t && t < cnt ? power(cnt - 1 - t) : 0.f;
    co[t * ST_ROW + ST_B + s] = s <= t ? power(t - s) * dots[t][s] : 0.f;
    if (s == 0) {
      co[t * ST_ROW + 16] = 0.f;
      co[t * ST_ROW + 17] = 1.f;
      co[t * ST_ROW + 18] = power(t + 1);
      co[t * ST_ROW + 19] = power(cnt);
    }
  }
}

template <int R>
__global__ void __launch_bounds__(ST_THREADS)
lightning_tiles_kernel(const float* __restrict__ proj, long long ld, int v_off, const float* __restrict__ qk,
                       const float* __restrict__ coef, float* __restrict__ state, long long state_stride,
                       const int* __restrict__ qo_indptr, const int* __restrict__ state_slots, float* __restrict__ out, int H, int dim,
                       int vdim, int act) {
  bspec::pdl_prologue_late(65);
  const int e = blockIdx.z, h = blockIdx.y;
  const int q_begin = qo_indptr[e], n = qo_indptr[e + 1] - q_begin;
  if (n < ST_FROM) return;
  StateTiles p;
  p.q = qk + ((size_t)q_begin * H + h) * 2 * dim, p.k = p.q + dim;
  p.q_stride = p.k_stride = (long long)H * 2 * dim;
  p.v = proj + (size_t)q_begin * ld + v_off + (size_t)h * vdim, p.v_stride = ld;
  p.coef = coef + (state_tile_slot(q_begin, e, 0) * H + h) * ST_CO, p.coef_stride = (long long)H * ST_CO;
  p.s = state + (size_t)state_slots[e] * state_stride + (size_t)h * vdim * dim, p.s_stride = p.s_rows = dim;
  p.out = out + (size_t)q_begin * H * vdim + (size_t)h * vdim, p.out_stride = (long long)H * vdim;
  p.n = n, p.dim = dim, p.vdim = vdim, p.j0 = blockIdx.x * ST_COLS;
  state_tiles<R, false>(p, [act](float x) { return act ? silu_f(x) : x; });
}

template <int R>
int launch_lightning_tiles(dim3 grid, cudaStream_t stream, const float* proj, long long ld, int v_off, const float* qk, const float* coef,
                           float* state, long long state_stride, const int* qo_indptr, const int* state_slots, float* out, int H,
                           int dim, int vdim, int act) {
  static bool set[bspec::kMaxDevices] = {};
  bool& done = set[bspec::current_device()];
  if (!done) {
    const cudaError_t err = cudaFuncSetAttribute(lightning_tiles_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)state_tiles_smem(16 * R));
    if (err != cudaSuccess) return (int)err;
    done = true;
  }
  BSPEC_LAUNCH_SERIALIZED((lightning_tiles_kernel<R>), grid, ST_THREADS, state_tiles_smem(16 * R), stream, proj, ld, v_off, qk, coef,
                          state, state_stride, qo_indptr, state_slots, out, H, dim, vdim, act);
  return BSPEC_LAUNCH_CHECK();
}

// ---------------------------------------------------------------- lightning attention, chunks at once
// With a fixed decay what a chunk of 64 tokens adds to S does not depend on S, so only the decayed sum over the chunks is a
// chain; everything else is products of whole chunks, formed by all SMs at once:
//   lightning_chunk_sums   U_c = sum_t d^(cnt-1-t) k_t v_t^T                    [value columns x key rows] per chunk and head
//   lightning_chunk_scan   S_c = d^cnt S_(c-1) + U_(c-1), over a head's chunks; S_c takes U_c's place
//   lightning_chunk_out    o_t = d^(t+1) S_c^T q_t + sum_(s <= t) d^(t-s) (q_t . k_s) v_s
// Float32 throughout, in packed multiply-adds; bound by them (3.1 million per chunk and head of 128 x 128).  q and k are
// prepared (activation, scale, rotation) where they are loaded: a kernel of its own for that took 25 us a layer at 2,048 tokens
// and 16 heads, and their memory.
constexpr long long CH_SCRATCH = 64ll << 20;         // floats of the chunks' sums at most
constexpr int CH_SUM_SMEM = 2 * CH * CH_W * 4;
constexpr int CH_OUT_SMEM = (2 * CH * CH_LD + CH * CH_AT + CH_W * (CH_SL + 4) + CH + 1) * 4;

// d^u, formed in float64
__device__ __forceinline__ float power_of(float d, int u) {
  double r = 1.0, b = d;
  for (; u > 0; u >>= 1, b *= b)
    if (u & 1) r *= b;
  return (float)r;
}

// A lane's quad of eight rows of a chunk (rows warp + 8 u, columns 4 lane ..): zeros past ``cnt`` and ``width``.
struct ChunkQuads {
  float4 v[CH / 8];
  __device__ __forceinline__ void load(const float* __restrict__ src, long long ld, int cnt, int width, bool vec) {
    const int c = 4 * (threadIdx.x & 31);
#pragma unroll
    for (int u = 0; u < CH / 8; ++u) {
      const int t = (threadIdx.x >> 5) + 8 * u;
      const float* p = src + (size_t)t * ld + c;
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < cnt && c < width) {
        if (vec) v[u] = *reinterpret_cast<const float4*>(p);
        else v[u] = make_float4(p[0], c + 1 < width ? p[1] : 0.f, c + 2 < width ? p[2] : 0.f, c + 3 < width ? p[3] : 0.f);
      }
    }
  }
  // to rows of ``lds`` floats; silu(0) = 0
  __device__ __forceinline__ void store(float* dst, int lds, int act, float scale) const {
#pragma unroll
    for (int u = 0; u < CH / 8; ++u) {
      float4 o = v[u];
      if (act) o = make_float4(silu_f(o.x), silu_f(o.y), silu_f(o.z), silu_f(o.w));
      *reinterpret_cast<float4*>(dst + ((threadIdx.x >> 5) + 8 * u) * lds + 4 * (threadIdx.x & 31)) =
          make_float4(o.x * scale, o.y * scale, o.z * scale, o.w * scale);
    }
  }
};
// The rotation of a chunk's prepared rows, in place.
template <int N>
__device__ __forceinline__ void chunk_rotate(float* const (&rows)[N], int lds, int cnt, const float* __restrict__ inv_freq, int rot,
                                             const int* __restrict__ positions) {
  const int half = rot / 2;
  for (int x = threadIdx.x; x < cnt * half; x += CH_THREADS) {
    const int t = x / half, d = x - t * half;
    float sn, c;
    rotation_sincos(positions[t], inv_freq, half, d, &sn, &c);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float* r = rows[i] + t * lds + d;
      const float u = r[0], v = r[half];
      r[0] = u * c - v * sn;
      r[half] = v * c + u * sn;
    }
  }
  __syncthreads();
}

// Block: one chunk and head; thread (tx, ty): rows 4 tx + {0..3} and 64 more, columns 4 ty + {0..3} and 64 more.
__global__ void __launch_bounds__(CH_THREADS, 2)
lightning_chunk_sums_kernel(const float* __restrict__ proj, long long ld, int k_off, int v_off, const float* __restrict__ decay,
                            const int* __restrict__ qo_indptr, int n_entries, float* __restrict__ sums, int H, int dim, int vdim, int act,
                            float k_scale, const float* __restrict__ inv_freq, int rot, const int* __restrict__ positions, int vec) {
  bspec::pdl_prologue(65);
  extern __shared__ __align__(16) float smem_f[];
  float *ks = smem_f, *vs = smem_f + CH * CH_W;
  __shared__ float pw[CH];                           // powers of the decay
  const int h = blockIdx.y, e = chunk_entry(qo_indptr, n_entries, blockIdx.x);
  const int q_begin = qo_indptr[e], n = qo_indptr[e + 1] - q_begin, i = blockIdx.x - (int)chunk_slot(q_begin, e, 0);
  if (n < ST_FROM || i * CH >= n) return;
  const int cnt = min(CH, n - i * CH), t0 = q_begin + i * CH, tid = threadIdx.x;
  if (tid < CH) pw[tid] = power_of(decay[h], tid);
  const float* first = proj + (size_t)t0 * ld;
  ChunkQuads k, v;
  k.load(first + k_off + (size_t)h * dim, ld, cnt, dim, vec);
  v.load(first + v_off + (size_t)h * vdim, ld, cnt, vdim, vec);
  __syncthreads();
  k.store(ks, CH_W, act, k_scale);
#pragma unroll
  for (int u = 0; u < CH / 8; ++u) {                 // the powers go to the values
    const int t = (tid >> 5) + 8 * u;
    const float p = pw[max(cnt - 1 - t, 0)];
    float4 o = v.v[u];
    if (act) o = make_float4(silu_f(o.x), silu_f(o.y), silu_f(o.z), silu_f(o.w));
    *reinterpret_cast<float4*>(vs + t * CH_W + 4 * (tid & 31)) = make_float4(p * o.x, p * o.y, p * o.z, p * o.w);
  }
  __syncthreads();
  if (rot > 0) {
    float* const rows[1] = {ks};
    chunk_rotate(rows, CH_W, cnt, inv_freq, rot, positions + t0);
  }
  const int tx = tid & 15, ty = tid >> 4;
  unsigned long long acc[4][8];                      // [pair of rows][column]
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[a][b] = 0ull;
#pragma unroll 2
  for (int t = 0; t < cnt; ++t) {
    const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(ks + t * CH_W + 4 * tx);
    const ulonglong2 k1 = *reinterpret_cast<const ulonglong2*>(ks + t * CH_W + 64 + 4 * tx);
    const float4 v0 = *reinterpret_cast<const float4*>(vs + t * CH_W + 4 * ty), v1 = *reinterpret_cast<const float4*>(vs + t * CH_W + 64 + 4 * ty);
    const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    const unsigned long long k[4] = {k0.x, k0.y, k1.x, k1.y};
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const unsigned long long vb = pair_of(v[b], v[b]);
#pragma unroll
      for (int a = 0; a < 4; ++a) fma_pair(acc[a][b], k[a], vb);
    }
  }
  float* dst = sums + ((size_t)blockIdx.x * H + h) * vdim * dim;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int j = (b < 4 ? 0 : 64) + 4 * ty + (b & 3);
    if (j >= vdim) continue;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int r = 64 * a + 4 * tx;
      if (r < dim) {
        float4 o;
        halves_of(acc[2 * a][b], o.x, o.y);
        halves_of(acc[2 * a + 1][b], o.z, o.w);
        *reinterpret_cast<float4*>(dst + (size_t)j * dim + r) = o;
      }
    }
  }
}

// A thread takes four numbers of one head's S through the chunks of a portion, eight chunks' sums asked for at a time; the blocks go
// over the requests, of which at most n / ST_FROM have chunks.  (One number per thread and blocks for every request: beside 31
// decoded requests of 64 heads 131,000 blocks: a step of 512 tokens and those 363 us, and 226 now.)
__global__ void __launch_bounds__(256)
lightning_chunk_scan_kernel(float* __restrict__ sums, const float* __restrict__ decay, float* __restrict__ state, long long state_stride,
                            const int* __restrict__ qo_indptr, const int* __restrict__ state_slots, int n_entries, int H, int numbers,
                            int vec) {
  bspec::pdl_prologue(65);
  const int h = blockIdx.y, x = 4 * (blockIdx.x * 256 + threadIdx.x);
  if (x >= numbers) return;
  const float d = decay[h], whole = power_of(d, CH);
  const size_t step = (size_t)H * numbers;
  for (int e = blockIdx.z; e < n_entries; e += gridDim.z) {
    const int q_begin = qo_indptr[e], n = qo_indptr[e + 1] - q_begin;
    if (n < ST_FROM) continue;
    const int chunks = (n + CH - 1) / CH;
    const float rest = power_of(d, n - (chunks - 1) * CH);
    float* sp = state + (size_t)state_slots[e] * state_stride + (size_t)h * numbers + x;
    float* up = sums + (chunk_slot(q_begin, e, 0) * H + h) * numbers + x;
    float4 s = vec ? *reinterpret_cast<const float4*>(sp) : make_float4(sp[0], sp[1], sp[2], sp[3]);
    for (int c0 = 0; c0 < chunks; c0 += 8) {
      float4 u[8];
#pragma unroll
      for (int c = 0; c < 8; ++c)
        u[c] = c0 + c < chunks ? *reinterpret_cast<const float4*>(up + (c0 + c) * step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c0 + c < chunks) {
          *reinterpret_cast<float4*>(up + (c0 + c) * step) = s;
          const float f = c0 + c == chunks - 1 ? rest : whole;
          s = make_float4(fmaf(f, s.x, u[c].x), fmaf(f, s.y, u[c].y), fmaf(f, s.z, u[c].z), fmaf(f, s.w, u[c].w));
        }
    }
    if (vec) *reinterpret_cast<float4*>(sp) = s;
    else sp[0] = s.x, sp[1] = s.y, sp[2] = s.z, sp[3] = s.w;
  }
}

// Block: one chunk and head, 64 tokens x 128 value columns.  First the chunk's own q . k (thread (tx, ty): tokens ty + 16 a
// against tx + 16 b), kept as at[s][t]; then per warp eight tokens, per lane columns lane + 32 b: S_c^T q over slices of 32 key
// rows, then the values' sum.
__global__ void __launch_bounds__(CH_THREADS, 2)
lightning_chunk_out_kernel(const float* __restrict__ proj, long long ld, int q_off, int k_off, int v_off, const float* __restrict__ decay,
                           const int* __restrict__ qo_indptr, int n_entries, const float* __restrict__ sums, float* __restrict__ out, int H,
                           int dim, int vdim, int act, float k_scale, const float* __restrict__ inv_freq, int rot,
                           const int* __restrict__ positions, int vec) {
  bspec::pdl_prologue(65);
  extern __shared__ __align__(16) float smem_f[];
  float* qs = smem_f;                                // [CH][CH_LD]
  float* kv = qs + CH * CH_LD;                       // [CH][CH_LD] k, then v
  float* at = kv + CH * CH_LD;                       // [CH s][CH_AT t]
  float* ss = at + CH * CH_AT;                       // [CH_W columns][CH_SL + 4 rows]
  float* pw = ss + CH_W * (CH_SL + 4);               // [CH + 1] powers of the decay
  const int h = blockIdx.y, e = chunk_entry(qo_indptr, n_entries, blockIdx.x);
  const int q_begin = qo_indptr[e], n = qo_indptr[e + 1] - q_begin, i = blockIdx.x - (int)chunk_slot(q_begin, e, 0);
  if (n < ST_FROM || i * CH >= n) return;
  const int cnt = min(CH, n - i * CH), t0 = q_begin + i * CH, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid <= CH) pw[tid] = power_of(decay[h], tid);
  const float* first = proj + (size_t)t0 * ld;
  {
    ChunkQuads q, k;
    q.load(first + q_off + (size_t)h * dim, ld, cnt, dim, vec);
    k.load(first + k_off + (size_t)h * dim, ld, cnt, dim, vec);
    q.store(qs, CH_LD, act, 1.f);
    k.store(kv, CH_LD, act, k_scale);
  }
  __syncthreads();
  if (rot > 0) {
    float* const rows[2] = {qs, kv};
    chunk_rotate(rows, CH_LD, cnt, inv_freq, rot, positions + t0);
  }
  {
    const int tx = tid & 15, ty = tid >> 4;
    unsigned long long acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = 0ull;
    for (int c = 0; c < dim; c += 4) {
      ulonglong2 q[4], k[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) q[a] = *reinterpret_cast<const ulonglong2*>(qs + (ty + 16 * a) * CH_LD + c);
#pragma unroll
      for (int b = 0; b < 4; ++b) k[b] = *reinterpret_cast<const ulonglong2*>(kv + (tx + 16 * b) * CH_LD + c);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          fma_pair(acc[a][b], q[a].x, k[b].x);
          fma_pair(acc[a][b], q[a].y, k[b].y);
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int t = ty + 16 * a, s = tx + 16 * b;
        float x, y;
        halves_of(acc[a][b], x, y);
        at[s * CH_AT + t] = s <= t ? pw[t - s] * (x + y) : 0.f;
      }
  }
  __syncthreads();                                   // everybody is done with k
  {
    ChunkQuads v;
    v.load(first + v_off + (size_t)h * vdim, ld, cnt, vdim, vec);
    v.store(kv, CH_LD, act, 1.f);
  }
  const float* S = sums + ((size_t)blockIdx.x * H + h) * vdim * dim;
  const int tb = 8 * warp;                           // this warp's tokens
  unsigned long long acc[8][4];
  chunk_read_state(acc, qs, ss, S, dim, vdim, tb, lane);
  bspec::pdl_launch_dependents();
  unsigned long long o[4][4];                        // [pair of tokens][column]
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      float x0, y0, x1, y1;
      halves_of(acc[2 * a][b], x0, y0);
      halves_of(acc[2 * a + 1][b], x1, y1);
      o[a][b] = pair_of(pw[tb + 2 * a + 1] * (x0 + y0), pw[tb + 2 * a + 2] * (x1 + y1));
    }
  chunk_below(o, at, tb, [&](int s, int b) { return kv[s * CH_LD + lane + 32 * b]; });
  chunk_write(o, out + ((size_t)t0 * H + h) * vdim, (long long)H * vdim, vdim, cnt, tb, lane);
}

// ---------------------------------------------------------------- selective scan
// xz [n, ld]: columns [x: inner | z: inner] of the in-projection.  State of a request at state + slot * stride:
// [N][inner] float32 (the scan's S, state index major), then at tail_off [(taps-1)][inner] the last inputs of the
// convolution, oldest first.  a2t [N][inner] float32: A[c, n] = -exp(A_log[c, n]), made once from the weights.

// xc[t, c] = silu(bias[c] + sum_j conv[c, j] * x[t - (taps-1) + j, c]); one thread per (token, channel).
template <typename T>
__global__ void __launch_bounds__(256)
scan_conv_kernel(const float* __restrict__ xz, long long ld, const void* __restrict__ conv, const void* __restrict__ bias,
                 int w_dtype, const float* __restrict__ state, long long state_stride, long long tail_off,
                 const int* __restrict__ qo_indptr, const int* __restrict__ tok_entry,
                 const int* __restrict__ state_slots, float* __restrict__ xc, T* __restrict__ xc_run, int inner,
                 int taps) {
  bspec::pdl_prologue(66);
  const int t = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= inner) return;
  const int e = tok_entry[t];
  const int i = t - qo_indptr[e];
  const float* tail = state + (size_t)state_slots[e] * state_stride + tail_off;
  float y = load_as_f32(bias, w_dtype, c);
  for (int j = 0; j < taps; ++j) {                           // oldest input first
    const int rel = i - (taps - 1 - j);
    const float x = rel >= 0 ? xz[(size_t)(t - (taps - 1 - j)) * ld + c] : tail[(size_t)(rel + taps - 1) * inner + c];
    y += load_as_f32(conv, w_dtype, (size_t)c * taps + j) * x;
  }
  const float v = silu_f(y);
  xc[(size_t)t * inner + c] = v;
  if (xc_run != nullptr) xc_run[(size_t)t * inner + c] = from_f32<T>(v);
}

// The same for four taps, with four channels and TT consecutive tokens per thread, for rows whose channels start on
// 16-byte boundaries: a thread keeps its weights and the last three inputs in registers.  Each channel's arithmetic is the
// same.
template <typename T, int TT>
__global__ void __launch_bounds__(256)
scan_conv4_kernel(const float* __restrict__ xz, long long ld, const float* __restrict__ conv, const float* __restrict__ bias,
                  const float* __restrict__ state, long long state_stride, long long tail_off,
                  const int* __restrict__ qo_indptr, const int* __restrict__ tok_entry,
                  const int* __restrict__ state_slots, float* __restrict__ xc, T* __restrict__ xc_run, int n, int inner) {
  bspec::pdl_prologue(66);
  const int t0 = blockIdx.x * TT;
  const int c = 4 * (blockIdx.y * blockDim.x + threadIdx.x);
  if (c >= inner) return;
  auto row4 = [](const float* p, float (&f)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  };
  float w[4][4], b[4], x[TT + 3][4];                         // x[u]: the input of token t0 + u - 3
#pragma unroll
  for (int q = 0; q < 4; ++q) row4(conv + (size_t)(c + q) * 4, w[q]);
  row4(bias + c, b);
#pragma unroll
  for (int u = 0; u < TT + 3; ++u) {
    const int t = t0 + u - 3;
#pragma unroll
    for (int q = 0; q < 4; ++q) x[u][q] = 0.f;
    if (t >= 0 && t < n) row4(xz + (size_t)t * ld + c, x[u]);
  }
#pragma unroll
  for (int u = 0; u < TT; ++u) {
    const int t = t0 + u;
    if (t >= n) break;
    const int e = tok_entry[t], i = t - qo_indptr[e];
    float y[4] = {b[0], b[1], b[2], b[3]};
#pragma unroll
    for (int j = 0; j < 4; ++j) {                            // oldest input first
      float v[4] = {x[u + j][0], x[u + j][1], x[u + j][2], x[u + j][3]};
      if (i < 3 - j) row4(state + (size_t)state_slots[e] * state_stride + tail_off + (size_t)(i + j) * inner + c, v);
#pragma unroll
      for (int q = 0; q < 4; ++q) y[q] += w[q][j] * v[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = silu_f(y[q]);
    *reinterpret_cast<float4*>(xc + (size_t)t * inner + c) = make_float4(y[0], y[1], y[2], y[3]);
    if (xc_run != nullptr)
#pragma unroll
      for (int q = 0; q < 4; ++q) xc_run[(size_t)t * inner + c + q] = from_f32<T>(y[q]);
  }
}

constexpr int SC_THREADS = 128;
constexpr int SC_TT = 8;
constexpr int SC_MAX_N = 256;

// LN lanes per channel; lane l keeps states l, l + LN, ... (NPL of them) of its channel in registers.  Tokens go
// SC_TT at a time: the next batch's B and C rows and the channel's own x, dt and z are fetched into registers while
// the recurrence runs over the current batch, and softplus and silu are taken once per batch outside the chain, so
// what is left per token is one exponential and two multiply-adds per state.  End to end, every token's arithmetic is the
// same wherever it falls in a batch, so the result does not depend on where a portion was cut.
//
// A chain of 2,048 tokens takes 605 us whatever the device has free (4,096 channels of 16 states: 32 to 128 blocks).  So
// long portions go in segments of SC_SEG tokens, all at once, where that is faster (bspec_scan_scratch): MODE 1 runs every segment from a zero state
// and leaves its end state and the sum of its dt; scan_segments_kernel carries the state from segment to segment,
// S <- exp(A sum dt) S + end, leaving the state before each; MODE 2 runs every segment again from there and writes the
// outputs.  Twice the arithmetic, but on all SMs.  MODE 0: the portion from end to end.
constexpr int SC_SEG = 64, SC_SEG_MIN = 512, SC_SEG_ENTRIES = 4, SC_SEG_MAX_N = 32;

// Where segment i of entry e has its state: segments of different entries never meet.
__device__ __forceinline__ size_t scan_segment_slot(int q_begin, int e, int i) { return (size_t)(q_begin / SC_SEG + e + i); }

template <typename T, int NPL, int LN, int MODE>
__global__ void __launch_bounds__(SC_THREADS)
selective_scan_kernel(const float* __restrict__ xz, long long ld, const float* __restrict__ xc,
                      const float* __restrict__ dt_raw, const float* __restrict__ bc, long long ld_bc,
                      const float* __restrict__ a2t, const void* __restrict__ dvec, const void* __restrict__ dt_bias,
                      int w_dtype, float* __restrict__ state, long long state_stride, long long tail_off,
                      const int* __restrict__ qo_indptr, const int* __restrict__ state_slots, T* __restrict__ out,
                      long long out_stride, float out_scale, int inner, int N, int taps, float* __restrict__ part,
                      float* __restrict__ dt_sum) {
  bspec::pdl_prologue_late(67);
  constexpr int NS = NPL * LN;                               // states this instance covers (N <= NS)
  constexpr int BCR = SC_TT * 2 * NS / SC_THREADS;           // staged B and C values per thread and batch
  static_assert(SC_TT * 2 * NS % SC_THREADS == 0, "the staged rows divide among the threads");
  __shared__ __align__(16) float bcs[SC_TT][2 * NS];         // [B: NS | C: NS] of a token, zeros beyond N
  const int e = blockIdx.y;
  const int lane = threadIdx.x % LN;
  const int c = blockIdx.x * (SC_THREADS / LN) + threadIdx.x / LN;
  const bool live = c < inner;
  const int cc = live ? c : 0;
  int t0 = qo_indptr[e], nt = qo_indptr[e + 1] - t0;
  float* sp = state + (size_t)state_slots[e] * state_stride;
  if constexpr (MODE != 0) {
    const int seg = blockIdx.z;
    if (seg * SC_SEG >= nt) return;
    const size_t slot = scan_segment_slot(t0, e, seg);
    sp = part + slot * N * inner;
    dt_sum += slot * inner;
    t0 += seg * SC_SEG;
    nt = min(SC_SEG, nt - seg * SC_SEG);
  }
  float total = 0.f;
  float xn[SC_TT], dn[SC_TT], zn[SC_TT], bn[BCR];
  auto fetch = [&](int base) {
    const int cnt = min(SC_TT, nt - base);
#pragma unroll
    for (int tt = 0; tt < SC_TT; ++tt) {
      if (tt >= cnt) break;
      const size_t t = (size_t)(t0 + base + tt);
      xn[tt] = xc[t * inner + cc];
      dn[tt] = dt_raw[t * inner + cc];
      zn[tt] = MODE == 1 ? 0.f : xz[t * ld + inner + cc];
    }
#pragma unroll
    for (int u = 0; u < BCR; ++u) {
      const int x = threadIdx.x + SC_THREADS * u;
      const int tt = x / (2 * NS), k = x % (2 * NS);
      const int n = k % NS;
      const bool ok = tt < cnt && n < N;
      bn[u] = ok ? bc[(size_t)(t0 + base + tt) * ld_bc + (k < NS ? n : N + n)] : 0.f;
    }
  };
  if (nt > 0) fetch(0);
  float s[NPL], a2[NPL];
#pragma unroll
  for (int m = 0; m < NPL; ++m) {
    const int n = lane + LN * m;
    const bool has = live && n < N;
    s[m] = has && MODE != 1 ? sp[(size_t)n * inner + cc] : 0.f;
    a2[m] = has ? a2t[(size_t)n * inner + cc] : 0.f;
  }
  const float dskip = load_as_f32(dvec, w_dtype, cc), dtb = load_as_f32(dt_bias, w_dtype, cc);
  for (int base = 0; base < nt; base += SC_TT) {
    const int cnt = min(SC_TT, nt - base);
    float xv[SC_TT], dv[SC_TT], gv[SC_TT];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < BCR; ++u) {
      const int x = threadIdx.x + SC_THREADS * u;
      bcs[x / (2 * NS)][x % (2 * NS)] = bn[u];
    }
#pragma unroll
    for (int tt = 0; tt < SC_TT; ++tt) {
      if (tt >= cnt) break;
      xv[tt] = xn[tt];
      dv[tt] = softplus_f(dn[tt] + dtb);
      if (MODE != 1) gv[tt] = silu_f(zn[tt]) * out_scale;
      if (MODE == 1) total += dv[tt];
    }
    __syncthreads();
    if (base + SC_TT < nt) fetch(base + SC_TT);
    // one token; the same arithmetic in a whole batch (unrolled without branches, so that the tokens' independent
    // work interleaves) and in a last, partial one
    auto token = [&](int tt, float xt, float dt, float gt) {
      const float dx = dt * xt;
      float y = 0.f;
      if constexpr (LN == 1 && NPL % 4 == 0) {
#pragma unroll
        for (int g = 0; g < NPL / 4; ++g) {
          const float4 b4 = *reinterpret_cast<const float4*>(&bcs[tt][4 * g]);
          const float4 c4 = *reinterpret_cast<const float4*>(&bcs[tt][NS + 4 * g]);
          const float bb[4] = {b4.x, b4.y, b4.z, b4.w}, cv[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            s[4 * g + q] = scan_update(s[4 * g + q], __fmul_rn(dt, a2[4 * g + q]), __fmul_rn(dx, bb[q]));
            y = __fmaf_rn(s[4 * g + q], cv[q], y);
          }
        }
      } else {
#pragma unroll
        for (int m = 0; m < NPL; ++m) {
          const int n = lane + LN * m;                       // states beyond N: a2 = 0, B = C = 0, s stays 0
          s[m] = scan_update(s[m], __fmul_rn(dt, a2[m]), __fmul_rn(dx, bcs[tt][n]));
          y = __fmaf_rn(s[m], bcs[tt][NS + n], y);
        }
      }
#pragma unroll
      for (int o = 1; o < LN; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      if (MODE != 1 && live && lane == 0)
        out[(size_t)(t0 + base + tt) * out_stride + cc] = from_f32<T>(__fmul_rn(__fmaf_rn(dskip, xt, y), gt));
    };
    if (cnt == SC_TT) {
#pragma unroll
      for (int tt = 0; tt < SC_TT; ++tt) token(tt, xv[tt], dv[tt], gv[tt]);
    } else {
#pragma unroll
      for (int tt = 0; tt < SC_TT; ++tt)
        if (tt < cnt) token(tt, xv[tt], dv[tt], gv[tt]);
    }
  }
  bspec::pdl_launch_dependents();
  if (!live || MODE == 2) return;
#pragma unroll
  for (int m = 0; m < NPL; ++m) {
    const int n = lane + LN * m;
    if (n < N) sp[(size_t)n * inner + cc] = s[m];
  }
  if (MODE == 1 && lane == 0) dt_sum[cc] = total;
  if (MODE == 0 && lane == 0) {
    // the convolution's last taps-1 inputs, oldest first: rows of this portion, and before them what the state held
    float* tail = sp + tail_off;
    for (int u = 0; u < taps - 1; ++u) {
      const int rel = nt - (taps - 1) + u;
      tail[(size_t)u * inner + cc] = rel >= 0 ? xz[(size_t)(t0 + rel) * ld + cc] : tail[(size_t)(u + nt) * inner + cc];
    }
  }
}

// One thread per (channel, state): the state carried over the portion's segments; part[segment] takes the state before it.
// A segment's exponent is the sum of its tokens': near zero, where 1 - exp(x) is what matters, the state moves by the small
// difference as in scan_update; where most of the state is gone, exp(x) S + end is the form without cancellation (s + (end - s)
// would leave a rounding of the state before, whole, in the state after).
// The blocks of state 0 also keep the convolution's last taps - 1 inputs.
__global__ void __launch_bounds__(128)
scan_segments_kernel(const float* __restrict__ xz, long long ld, const float* __restrict__ a2t, float* __restrict__ state,
                     long long state_stride, long long tail_off, const int* __restrict__ qo_indptr,
                     const int* __restrict__ state_slots, int inner, int N, int taps, float* __restrict__ part,
                     const float* __restrict__ dt_sum) {
  bspec::pdl_prologue(67);
  const int e = blockIdx.z, n = blockIdx.y, c = blockIdx.x * 128 + threadIdx.x;
  const int t0 = qo_indptr[e], nt = qo_indptr[e + 1] - t0;
  if (c >= inner || nt <= 0) return;
  float* sp = state + (size_t)state_slots[e] * state_stride;
  const int segs = (nt + SC_SEG - 1) / SC_SEG;
  const size_t first = scan_segment_slot(t0, e, 0), step = (size_t)N * inner;
  float* pp = part + first * step + (size_t)n * inner + c;
  const float* dp = dt_sum + first * inner + c;
  const float a2 = a2t[(size_t)n * inner + c];
  float s = sp[(size_t)n * inner + c];
  for (int i0 = 0; i0 < segs; i0 += 8) {                       // eight segments' numbers asked for at a time
    float end[8], dts[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool ok = i0 + u < segs;
      end[u] = ok ? pp[(i0 + u) * step] : 0.f;
      dts[u] = ok ? dp[(size_t)(i0 + u) * inner] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + u < segs) {
        pp[(i0 + u) * step] = s;
        const float x = __fmul_rn(dts[u], a2);
        s = x > -0.5f ? scan_update(s, x, end[u]) : __fmaf_rn(expf(x), s, end[u]);
      }
  }
  sp[(size_t)n * inner + c] = s;
  if (n == 0) {
    float* tail = sp + tail_off;
    for (int u = 0; u < taps - 1; ++u) {
      const int rel = nt - (taps - 1) + u;
      tail[(size_t)u * inner + c] = rel >= 0 ? xz[(size_t)(t0 + rel) * ld + c] : tail[(size_t)(u + nt) * inner + c];
    }
  }
}
}  // namespace

// How the portions of ST_FROM tokens and more of a step of n tokens in portions of min_q_len to max_q_len go: 0 token by token,
// 1 by tiles, 2 by chunks.  Chunks where tiles pay, the heads fill most of the 128 x 128 numbers that a chunk's products are
// laid out for, and an estimate of both says so.  Tiles: the longest portion's chain, slower where an SM holds two heads' blocks, or
// the work of a full device, to the last of its blocks' rounds.  Chunks: the products of all chunks, partial ones like whole ones,
// and every further portion's states.  Fitted to 160 steps (1 to 64 heads of 96 to 128, 1 to 101 requests); the choice is at most 3 %
// slower than tiles, and leaves up to 17 % in a few steps of several portions.  Tiles / chunks, us, heads of 128 x 128:
//   16 heads: 512 66 / 67; 1,000 124 / 74; 2,048 254 / 144; 2,048 beside 31 decoded 360 / 167; eight of 600 391 / 388; 512 beside twenty
//   of 64 142 / 178; 2,048 beside twenty of 200 460 / 582; 520 beside a hundred of 70 590 / 1,484
//   4 heads: 512 63 / 56; 2,048 231 / 73; 512 beside twenty of 64 74 / 73; 520 beside a hundred of 70 163 / 302
//   64 heads: 512 207 / 143; 2,048 724 / 575; 512 beside four of 300 498 / 558; 512 beside twenty of 64 522 / 953
//   16 heads of 96 x 96: 512 65 / 81; 1,000 122 / 84; three of 512 98 / 134; 32 of 512 876 / 1,223
static int lightning_form(int n, int n_entries, int min_q_len, int max_q_len, int H, int dim, int vdim) {
  if (n <= 0 || n_entries <= 0 || H <= 0 || dim <= 0 || vdim <= 0) return 0;
  // (the token loop's time per unit of work falls with the blocks that share the device)
  const long long blocks = (long long)((vdim + LT_COLS - 1) / LT_COLS) * H * n_entries, sms = bspec::sm_count();
  const double rate = (blocks < 3 * sms ? 1.0e-6 : (blocks < 6 * sms ? 0.66e-6 : 0.45e-6)) * (dim <= 32 ? 1.42 : 1.0);
  const bspec::TokenCost tokens = {dim <= 32 ? 0.165 : (dim <= 64 ? 0.19 : (dim <= 128 ? 0.25 : 0.38)), rate};
  const bspec::TokenCost tiles = {dim <= 128 ? 0.115 : 0.165, dim <= 128 ? 6.0e-4 : 9e-4};
  if (!bspec::tiles_pay(n, n_entries, min_q_len, max_q_len, H, dim, vdim, tokens, tiles)) return 0;
  if (max_q_len < CH_FROM || !chunk_sizes(dim, vdim) || chunk_slots(n, n_entries) * H * dim * vdim > CH_SCRATCH) return 1;
  const bspec::Tall t = bspec::tall_portions(n, n_entries, min_q_len, max_q_len);
  const double per = (double)((vdim + LT_COLS - 1) / LT_COLS) * H, all = per * t.count;        // blocks of a portion, of all
  const double rounds = all < 4.0 * sms ? (double)(((long long)all + sms - 1) / sms * sms) / all : 1.0;
  const double by_tiles = max(max_q_len * (all <= sms ? 0.118 : 0.175), t.tokens * per * 5.5e-4 * rounds) +
                          t.tokens * H * (0.5e-4 + 2e-6 * dim) + 7.5;
  const double parts = ((max_q_len + CH - 1) / CH + (t.tokens - max_q_len) / CH + 0.5 * (t.count - 1)) * H;
  const bool whole = dim == CH_W && vdim == CH_W;
  const double by_chunks = max((whole ? 48.0 : 70.0) + 0.1 * parts, (whole ? 0.27 : 0.31) * parts) + 0.33 * (t.count - 1) * H;
  return by_chunks < 0.96 * by_tiles ? 2 : 1;
}

// Floats of scratch: the tiles' coefficients with prepared q and k (as large as the step's q and k columns), or the chunks' sums;
// 0 where no portion goes by either.
BSPEC_API long long bspec_lightning_scratch(int n, int n_entries, int min_q_len, int max_q_len, int H, int dim, int vdim) {
  const int form = lightning_form(n, n_entries, min_q_len, max_q_len, H, dim, vdim);
  if (form == 0) return 0;
  return form == 2 ? chunk_slots(n, n_entries) * H * dim * vdim : (long long)n * H * 2 * dim + bspec::state_tile_slots(n, n_entries) * H * ST_CO;
}
// Kernels that a step launches.
BSPEC_API int bspec_lightning_launches(int n, int n_entries, int min_q_len, int max_q_len, int H, int dim, int vdim) {
  const int form = lightning_form(n, n_entries, min_q_len, max_q_len, H, dim, vdim);
  return form == 0 ? 1 : (form == 2 ? 3 : 2) + (min_q_len < ST_FROM ? 1 : 0);
}

BSPEC_API int bspec_lightning_recurrence(const float* proj, long long ld, int q_off, int k_off, int v_off,
                                         const float* decay, float* state, long long state_stride,
                                         const int* qo_indptr, const int* state_slots, float* out, int n, int n_entries,
                                         int min_q_len, int max_q_len, int H, int dim, int vdim, int act, float k_scale,
                                         const float* inv_freq, int rot, const int* positions, float* scratch,
                                         cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (rot < 0 || rot > dim || rot % 2 || (rot > 0 && (inv_freq == nullptr || positions == nullptr)))
    return (int)cudaErrorInvalidValue;
  if (dim <= 0 || dim > 256 || vdim <= 0 || H <= 0 || H > 65535 || n_entries > 65535)
    return (int)cudaErrorInvalidValue;
  const int form = scratch != nullptr ? lightning_form(n, n_entries, min_q_len, max_q_len, H, dim, vdim) : 0;
  if (form == 2) {
    const int vec = ((ld | q_off | k_off | v_off | dim | vdim) & 3) == 0 && ((uintptr_t)proj & 15) == 0;
    static bool set[bspec::kMaxDevices] = {};
    bool& done = set[bspec::current_device()];
    if (!done) {
      cudaError_t e = cudaFuncSetAttribute(lightning_chunk_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CH_SUM_SMEM);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(lightning_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CH_OUT_SMEM);
      if (e != cudaSuccess) return (int)e;
      done = true;
    }
    const dim3 chunks((unsigned)chunk_slots(n, n_entries), H);
    BSPEC_LAUNCH(lightning_chunk_sums_kernel, chunks, CH_THREADS, CH_SUM_SMEM, stream, proj, ld, k_off, v_off, decay, qo_indptr, n_entries,
                 scratch, H, dim, vdim, act, k_scale, inv_freq, rot, positions, vec);
    BSPEC_LAUNCH(lightning_chunk_scan_kernel, dim3((dim * vdim + 1023) / 1024, H, min(n_entries, n / ST_FROM)), 256, 0, stream, scratch,
                 decay, state, state_stride, qo_indptr, state_slots, n_entries, H, dim * vdim,
                 (int)(state_stride % 4 == 0 && ((uintptr_t)state & 15) == 0));
    BSPEC_LAUNCH(lightning_chunk_out_kernel, chunks, CH_THREADS, CH_OUT_SMEM, stream, proj, ld, q_off, k_off, v_off, decay, qo_indptr,
                 n_entries, (const float*)scratch, out, H, dim, vdim, act, k_scale, inv_freq, rot, positions, vec);
    const int err = BSPEC_LAUNCH_CHECK();
    if (err != 0 || min_q_len >= ST_FROM) return err;
  }
  if (form == 1) {
    float* qk = scratch + bspec::state_tile_slots(n, n_entries) * H * ST_CO;
    BSPEC_LAUNCH(lightning_tiles_prepare_kernel, dim3((unsigned)bspec::state_tile_slots(n, n_entries), H), 128, 0, stream, proj, ld,
                 q_off, k_off, decay, qo_indptr, n_entries, qk, scratch, H, dim, act, k_scale, inv_freq, rot, positions);
    const int err = BSPEC_LAUNCH_CHECK();
    if (err != 0) return err;
    const dim3 tiles((vdim + ST_COLS - 1) / ST_COLS, H, n_entries);
    const int tiled = dim <= 128 ? launch_lightning_tiles<8>(tiles, stream, proj, ld, v_off, qk, scratch, state, state_stride, qo_indptr,
                                                  state_slots, out, H, dim, vdim, act)
                      : launch_lightning_tiles<16>(tiles, stream, proj, ld, v_off, qk, scratch, state, state_stride, qo_indptr,
                                                  state_slots, out, H, dim, vdim, act);
    if (tiled != 0 || min_q_len >= ST_FROM) return tiled;
  }
  const int below = form != 0 ? ST_FROM : 0x7fffffff;           // the portions left for the token loop
  const dim3 grid((vdim + LT_COLS - 1) / LT_COLS, H, n_entries);
  // few blocks (a lone prompt): 32 lanes per column, so that an SM holds 16 warps of its one block; many blocks
  // (a decode batch): 8 lanes with more rows each, and the SMs fill with blocks
  const bool few = (long long)grid.x * grid.y * grid.z < 4 * 148;
#define LL(NR, L)                                                                                                  \
  BSPEC_LAUNCH_SERIALIZED((lightning_recurrence_kernel<NR, L>), grid, LT_COLS * L, 0, stream, proj, ld, q_off,     \
                          k_off, v_off, decay, state, state_stride, qo_indptr, state_slots, out, H, dim, vdim, act,   \
                          k_scale, inv_freq, rot, positions, below)
  if (dim <= 32) LL(4, 8);
  else if (dim <= 64) { if (few) LL(4, 16); else LL(8, 8); }
  else if (dim <= 128) { if (few) LL(4, 32); else LL(16, 8); }
  else { if (few) LL(8, 32); else LL(32, 8); }
#undef LL
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_API int bspec_scan_conv(const float* xz, long long ld, const void* conv, const void* bias, int w_dtype,
                              const float* state, long long state_stride, long long tail_off, const int* qo_indptr,
                              const int* tok_entry, const int* state_slots, float* xc, void* xc_run, int run_dtype,
                              int n, int inner, int taps, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (inner <= 0 || taps < 1) return (int)cudaErrorInvalidValue;
  if (taps == 4 && inner % 4 == 0 && ld % 4 == 0 && tail_off % 4 == 0 && state_stride % 4 == 0 && w_dtype == BSPEC_F32 &&
      ((reinterpret_cast<uintptr_t>(xz) | reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(bias) |
        reinterpret_cast<uintptr_t>(conv) | reinterpret_cast<uintptr_t>(xc)) & 15) == 0) {
    const int quads = inner / 4, per = quads >= 128 ? 128 : ((quads + 31) / 32) * 32;
    const bool many = (long long)n * quads >= 1ll << 20;     // a prompt: enough threads also with eight tokens each
    const dim3 grid4(many ? (n + 7) / 8 : n, (quads + per - 1) / per);
    if (grid4.y > 65535) return (int)cudaErrorInvalidConfiguration;
#define LC(T, TT) BSPEC_LAUNCH((scan_conv4_kernel<T, TT>), grid4, per, 0, stream, xz, ld, (const float*)conv, (const float*)bias, state, \
                               state_stride, tail_off, qo_indptr, tok_entry, state_slots, xc, \
                               run_dtype == BSPEC_F32 ? (T*)nullptr : (T*)xc_run, n, inner)
    if (run_dtype == BSPEC_F32) { if (many) LC(float, 8); else LC(float, 1); }
    else { if (many) LC(__nv_bfloat16, 8); else LC(__nv_bfloat16, 1); }
#undef LC
    return BSPEC_LAUNCH_CHECK();
  }
  const int threads = inner >= 256 ? 256 : ((inner + 31) / 32) * 32;
  const dim3 grid(n, (inner + threads - 1) / threads);
  if (grid.y > 65535) return (int)cudaErrorInvalidConfiguration;
  if (run_dtype == BSPEC_F32)
    BSPEC_LAUNCH((scan_conv_kernel<float>), grid, threads, 0, stream, xz, ld, conv, bias, w_dtype, state, state_stride,
                 tail_off, qo_indptr, tok_entry, state_slots, xc, (float*)nullptr, inner, taps);
  else
    BSPEC_LAUNCH((scan_conv_kernel<__nv_bfloat16>), grid, threads, 0, stream, xz, ld, conv, bias, w_dtype, state,
                 state_stride, tail_off, qo_indptr, tok_entry, state_slots, xc, (__nv_bfloat16*)xc_run, inner, taps);
  return BSPEC_LAUNCH_CHECK();
}

// Few channels x requests: more lanes per channel, so that a lone prompt's chain is shorter and more SMs take part.
static bool scan_few(int inner, int n_entries) { return (long long)((inner + SC_THREADS - 1) / SC_THREADS) * n_entries < 148; }

// Floats of scratch for a step of n tokens: 0 where the portions go from end to end.  In segments where the longest chain is
// long and twice the arithmetic spread over the device takes less time than that chain.  Both are estimated, us on a B200: end
// to end a chain whose tokens take longer the more blocks work beside it (those of n / max_q_len requests), in segments the work.
// Measured, end to end / in segments: 4,096 channels of 16 states 1 x 256 tokens 83 / 91, 1 x 2,048 599 / 254, 4 x 512 276 / 254;
// 8,192 channels 2 x 512 276 / 254, 3 x 512 340 / 359, 4 x 2,048 1,347 / 1,734, 2,048 tokens beside 3 1,337 / 482; 16,384 channels 1 x 512
// 277 / 255, 2 x 512 340 / 460; 4,096 channels of 32 states 1 x 512 213 / 145, 2 x 512 233 / 308; 8,192 1 x 512 233 / 314.  More than
// 32 states spread over several lanes of a channel and go from end to end.
BSPEC_API long long bspec_scan_scratch(int n, int n_entries, int max_q_len, int inner, int N) {
  if (max_q_len < SC_SEG_MIN || n_entries > SC_SEG_ENTRIES || N > SC_SEG_MAX_N) return 0;
  const double blocks = (double)((inner + SC_THREADS - 1) / SC_THREADS) * n / max_q_len, million = 1e-6 * n * inner;
  double token;
  if (scan_few(inner, n_entries)) {
    const double x = blocks > 32 ? blocks - 32 : 0;
    token = N <= 16 ? 0.29 * (1 + 0.0055 * x + 3e-5 * x * x) : 0.412 * (1 + 0.0003 * x + 8e-5 * x * x);
  } else {
    token = (N <= 16 ? 0.655 : 1.07) * (blocks > 300 ? blocks / 300 : 1);
  }
  if ((N <= 16 ? 50 + 25.2 * million : 30 + 55 * million) >= max_q_len * token) return 0;
  return (long long)(n / SC_SEG + n_entries + 1) * (N + 1) * inner;
}

BSPEC_API int bspec_selective_scan(const float* xz, long long ld, const float* xc, const float* dt_raw, const float* bc,
                                   long long ld_bc, const float* a2t, const void* dvec, const void* dt_bias,
                                   int w_dtype, float* state, long long state_stride, long long tail_off,
                                   const int* qo_indptr, const int* state_slots, void* out, int out_dtype,
                                   long long out_stride, float out_scale, int n, int n_entries, int max_q_len, int inner,
                                   int N, int taps, float* scratch, cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (inner <= 0 || N <= 0 || N > SC_MAX_N || taps < 1 || n_entries > 65535) return (int)cudaErrorInvalidValue;
  const bool few = scratch == nullptr && scan_few(inner, n_entries);
  const int segs = scratch != nullptr ? (max_q_len + SC_SEG - 1) / SC_SEG : 1;
  if (segs > 65535) return (int)cudaErrorInvalidConfiguration;
  float* dt_sum = scratch != nullptr ? scratch + (size_t)(n / SC_SEG + n_entries + 1) * N * inner : nullptr;
#define LSM(T, NPL, LN, MODE)                                                                                        \
  BSPEC_LAUNCH_SERIALIZED((selective_scan_kernel<T, NPL, LN, MODE>),                                                 \
                          dim3((inner + SC_THREADS / LN - 1) / (SC_THREADS / LN), n_entries, segs), SC_THREADS, 0,   \
                          stream, xz, ld, xc, dt_raw, bc, ld_bc, a2t, dvec, dt_bias, w_dtype, state, state_stride,   \
                          tail_off, qo_indptr, state_slots, (T*)out, out_stride, out_scale, inner, N, taps, scratch, \
                          dt_sum)
#define LS(T, NPL, LN) LSM(T, NPL, LN, 0)
#define LSS(T, NPL)                                                                                                  \
  do {                                                                                                               \
    LSM(float, NPL, 1, 1);                                                                                           \
    BSPEC_LAUNCH(scan_segments_kernel, dim3((inner + 127) / 128, N, n_entries), 128, 0, stream, xz, ld, a2t, state,  \
                 state_stride, tail_off, qo_indptr, state_slots, inner, N, taps, scratch, dt_sum);                   \
    LSM(T, NPL, 1, 2);                                                                                               \
  } while (0)
#define LSN(T)                                                                                                       \
  do {                                                                                                               \
    if (scratch != nullptr) {                                                                                        \
      if (N <= 16) LSS(T, 16); else LSS(T, 32);                                                                      \
    } else if (few) {                                                                                                \
      if (N <= 16) LS(T, 4, 4); else if (N <= 32) LS(T, 8, 4); else if (N <= 64) LS(T, 8, 8);                        \
      else if (N <= 128) LS(T, 16, 8); else LS(T, 32, 8);                                                            \
    } else {                                                                                                         \
      if (N <= 16) LS(T, 16, 1); else if (N <= 32) LS(T, 32, 1); else if (N <= 64) LS(T, 32, 2);                     \
      else if (N <= 128) LS(T, 32, 4); else LS(T, 32, 8);                                                            \
    }                                                                                                                \
  } while (0)
  if (out_dtype == BSPEC_F32) LSN(float); else LSN(__nv_bfloat16);
#undef LSN
#undef LS
#undef LSS
#undef LSM
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_DEFINE_TRACE_SETTER(bspec_trace_set_state_mixers)
BSPEC_DEFINE_BOUNDS_REPORT(bspec_bounds_report_state_mixers)
