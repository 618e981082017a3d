// True float32 matrix product on the CUDA cores (fused multiply-adds of float32 numbers, no tensor-core or
// reduced-precision mode):  C[M,N] = A[M,K] * W[N,K]^T, all row-major, K contiguous.
//
// The order of every sum is fixed by K alone, so that a row's bits do not depend on M, on the other rows of the batch or
// on the kernel that forms it:
//   slice   64 k:  one chain of fused multiply-adds over the even k and one over the odd k, in order, then their sum;
//   group   1,024 k: its slices, added in order;
//   result  the groups, added in order.
// (Even and odd k are the halves of Blackwell's packed fma.rn.f32x2, whose operands then are neighbours in memory.)
//
// Two kernels:
//   sgemm_rows_kernel  few rows (decode steps): bound by reading W once.  W streams through a ring of shared-memory
//                      stages by bulk copies, a thread owns one output number and one slice at a time.
//   sgemm_tile_kernel  everything else: bound by the multiply-adds.  BM x 64 tiles, 8 x 4 outputs per thread; 32 x 32 tiles
//                      where those would leave most of the device idle.
#include "tma.cuh"

using namespace bspec;

namespace {

constexpr int SLICE = 64, GROUP = 1024;

// the slice's value: its even chain plus its odd chain
__device__ __forceinline__ float fold2(unsigned long long acc) {
  float lo, hi;
  halves_of(acc, lo, hi);
  return lo + hi;
}

// named barrier of the consumer threads that also gives all of them the conjunction of ``ok``
__device__ __forceinline__ bool sync_and(bool ok) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, 64, p;\n\t"
      "selp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"((int)ok) : "memory");
  return r != 0;
}

// ------------------------------------------------------------------------------------------------ tiles
// A thread holds rows tm + (BM/8) i and columns tn + 16 j, TI x TJ = 8 x 4 outputs (32 x 32 tiles: 4 x 2 on 128 threads).  Both operands lie K-major in shared memory as
// they do in global memory (rows of 32 k and 4 floats of padding): a 16-byte load is two packed operands and nothing is
// transposed or duplicated.  A warp is 8 x 4 threads, placed so that neighbours share a row of A and neighbours of
// neighbours a row of W: both loads then take two passes of shared memory instead of four.  The group's running sum waits
// in shared memory, which keeps a thread at 128 registers and two blocks of 256 threads on an SM.
// Bound by the arithmetic.  968 x 16,384 x 2,048 on a B200: 1,684 us, 38.6 TFLOP/s (64 x 64 tiles of scalar multiply-adds
// with synchronous loads before: about 14.6 in a whole prompt); 8 x 8 outputs per thread and one block per SM: 1,784 us;
// scalar multiply-adds instead of packed ones: 2,047 us.
constexpr int BK = 32, LDT = BK + 4;

template <int BM> struct Tile {
  static constexpr int TI = BM == 32 ? 4 : 8, TJ = BM == 32 ? 2 : 4, BN = 16 * TJ, RM = BM / TI, NT = 16 * RM;
  static constexpr int SMEM = (2 * (BM + BN) * LDT + BM * BN) * 4, PER_SM = BM == 128 ? 2 : 4;
};

// 16 (VEC) or 4 bytes from global to shared memory, zeros where ``ok`` is false
template <bool VEC>
__device__ __forceinline__ void copy_or_zero(float* dst, const float* src, bool ok) {
  if constexpr (VEC)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s32(dst)), "l"(src), "r"(ok ? 4 : 0) : "memory");
}

// VEC: rows and pointers are multiples of 16 bytes.  grid (column tiles, row tiles, batch x splits): split s works on
// groups s, s + 1, .. of its share; with ``splits`` > 1 group g leaves its sum in part[(z * groups + g) * M * N], which
// sgemm_join_kernel adds up, else C takes the groups one after the other.
template <int BM, bool VEC>
__global__ void __launch_bounds__(Tile<BM>::NT, Tile<BM>::PER_SM)
sgemm_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, float* __restrict__ part,
                  int M, int N, int K, long long lda, long long ldw, long long ldc, long long sa, long long sw, long long sc,
                  int splits) {
  bspec::pdl_prologue(10);
  extern __shared__ __align__(16) float smem_f[];
  constexpr int NT = Tile<BM>::NT, RM = Tile<BM>::RM, BN = Tile<BM>::BN, TI = Tile<BM>::TI, TJ = Tile<BM>::TJ;
  float* as = smem_f;                               // [2][BM][LDT]
  float* ws = as + 2 * BM * LDT;                    // [2][BN][LDT]
  float* gsum = ws + 2 * BN * LDT;                  // [TI][NT][TJ]: outputs (i, 0 .. TJ - 1) of every thread at row i
  const int z = blockIdx.z / splits, split = blockIdx.z % splits;
  A += (size_t)z * sa;
  W += (size_t)z * sw;
  C += (size_t)z * sc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tm = (warp / 4) * 8 + ((lane >> 1) & 1) + 2 * (lane >> 3), tn = (warp & 3) * 4 + (lane & 1) + ((lane >> 1) & 2);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (K <= 0) {                                      // the empty sum
    for (int i = tid; i < BM * BN; i += NT)
      if (m0 + i / BN < M && n0 + i % BN < N) C[(size_t)(m0 + i / BN) * ldc + n0 + i % BN] = 0.f;
    return;
  }
  const int groups = (K + GROUP - 1) / GROUP, per = (groups + splits - 1) / splits;
  const int g_begin = split * per, g_end = min(groups, g_begin + per);
  const int t_begin = g_begin * (GROUP / BK), t_end = min((K + BK - 1) / BK, g_end * (GROUP / BK));

  // Every copy of a thread has the same k inside a stage; its rows are RS apart.  Rows past the operand's last are left
  // as they are: their outputs are not stored.  k past K become zeros.
  constexpr int WIDE = VEC ? 4 : 1, PER_ROW = BK / WIDE, RS = NT / PER_ROW, NA = BM / RS, NW = BN / RS;
  const int r0 = tid / PER_ROW, c0 = tid % PER_ROW * WIDE;
  const float* a_src = A + (size_t)(m0 + r0) * lda + c0;
  const float* w_src = W + (size_t)(n0 + r0) * ldw + c0;
  const long long a_step = RS * lda, w_step = RS * ldw;
  const int a_rows = (M - m0 - r0 + RS - 1) / RS, w_rows = (N - n0 - r0 + RS - 1) / RS;      // how many of the rows exist
  auto load = [&](int t, int buf) {
    const int k0 = t * BK;
    const bool ok = k0 + c0 < K;
    const float* ap = ok ? a_src + k0 : A;
    const float* wp = ok ? w_src + k0 : W;
    float* ad = as + (size_t)(buf * BM + r0) * LDT + c0;
    float* wd = ws + (size_t)(buf * BN + r0) * LDT + c0;
    const long long as_ = ok ? a_step : 0, ws_ = ok ? w_step : 0;
#pragma unroll
    for (int i = 0; i < NA; ++i)
      if (i < a_rows) copy_or_zero<VEC>(ad + i * RS * LDT, ap + i * as_, ok);
#pragma unroll
    for (int i = 0; i < NW; ++i)
      if (i < w_rows) copy_or_zero<VEC>(wd + i * RS * LDT, wp + i * ws_, ok);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  unsigned long long acc[TI][TJ];
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < TJ; ++j) acc[i][j] = 0ull;
  if (t_begin < t_end) load(t_begin, 0);
  for (int t = t_begin; t < t_end; ++t) {
    const int buf = (t - t_begin) & 1;
    if (t + 1 < t_end) {
      load(t + 1, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* a_ = as + (size_t)(buf * BM + tm) * LDT;
    const float* w_ = ws + (size_t)(buf * BN + tn) * LDT;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 b[TJ];
#pragma unroll
      for (int j = 0; j < TJ; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(w_ + 16 * j * LDT + k);
#pragma unroll
      for (int i = 0; i < TI; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_ + RM * i * LDT + k);
#pragma unroll
        for (int j = 0; j < TJ; ++j) fma_pair(acc[i][j], a.x, b[j].x);
#pragma unroll
        for (int j = 0; j < TJ; ++j) fma_pair(acc[i][j], a.y, b[j].y);
      }
    }
    const int done = (t + 1) * BK;
    if (done % SLICE == 0 || t + 1 == t_end) {
      const bool first = (t * BK) % GROUP < SLICE;                    // the group's first slice
#pragma unroll
      for (int i = 0; i < TI; ++i) {
        unsigned long long* q = acc[i];
        if constexpr (TJ == 4) {
          float4* at = reinterpret_cast<float4*>(gsum) + i * NT + tid;
          float4 v = make_float4(fold2(q[0]), fold2(q[1]), fold2(q[2]), fold2(q[3]));
          if (!first) {
            const float4 o = *at;
            v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
          }
          *at = v;
        } else {
          float2* at = reinterpret_cast<float2*>(gsum) + i * NT + tid;
          float2 v = make_float2(fold2(q[0]), fold2(q[1]));
          if (!first) {
            const float2 o = *at;
            v = make_float2(o.x + v.x, o.y + v.y);
          }
          *at = v;
        }
#pragma unroll
        for (int j = 0; j < TJ; ++j) q[j] = 0ull;
      }
      if (done % GROUP == 0 || t + 1 == t_end) {
        __syncthreads();
        const int g = t * BK / GROUP;
        float* dst = splits > 1 ? part + ((size_t)z * groups + g) * M * N : C;
        const long long ld = splits > 1 ? N : ldc;
        const bool set = splits > 1 || g == 0;
        for (int i = tid; i < BM * BN; i += NT) {
          const int m = m0 + i / BN, n = n0 + i % BN;
          if (m < M && n < N) {
            float* at = dst + (size_t)m * ld + n;
            // the output's place: row index ri of thread row tmi, column index cj of thread column tni
            const int ri = (i / BN) / RM, tmi = (i / BN) % RM, cj = (i % BN) / 16, tni = i % 16;
            const int owner = (tmi / 8 * 4 + tni / 4) * 32 + (tni & 1) + (tni & 2) * 2 + (tmi & 1) * 2 + (tmi & 6) * 4;
            const float v = gsum[(ri * NT + owner) * TJ + cj];
            *at = set ? v : *at + v;
          }
        }
      }
    }
    __syncthreads();
  }
}

// C = the groups' sums, added in order
__global__ void __launch_bounds__(256)
sgemm_join_kernel(const float* __restrict__ part, float* __restrict__ C, int M, int N, long long ldc, long long sc, int groups) {
  bspec::pdl_prologue(10);
  const long long mn = (long long)M * N;
  const float* p = part + (size_t)blockIdx.y * groups * mn;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < mn; i += (long long)gridDim.x * 256) {
    float v = p[i];
    for (int g = 1; g < groups; ++g) v += p[(size_t)g * mn + i];
    C[(size_t)blockIdx.y * sc + (size_t)(i / N) * ldc + i % N] = v;
  }
}

// ------------------------------------------------------------------------------------------------ few rows
// A block owns tiles of 16 rows of W (16 output numbers of MT tokens) one after the other; a stage is 512 k of them and of
// the tokens, fetched by a producer warp that runs ahead across tiles and, where W is a parameter (``w_ahead``: nothing on the
// stream before this kernel writes it), ahead of the end of the kernel before: W by one
// bulk copy per row, the tokens by 16-byte copies (a bulk copy costs an SM about 40 clocks whatever its size, which bound
// the kernel when the tokens' 256-byte slices were such copies: 347 us against 20x at 128,256 x 2,048 and 8 tokens).  Rows
// and slices are padded by 4 floats: a quarter warp's 16-byte loads fall into different banks.  64 consumer threads:
// rows tid % 8 and tid % 8 + 8, slice tid / 8 of the stage; two rows per thread halve the loads of the tokens' numbers,
// which bound the kernel at 8 tokens.  Two blocks per SM keep at least 128 KB of W in flight on an SM; where there are
// fewer tiles than SMs (``deep``), one block keeps that much.  4 tokens, us, two stages / five: 2,048 x 8,192 24.9 / 21.1, 2,048 x 16,384
// 47.1 / 39.7, 1,024 x 4,096 12.5 / 10.8; 8 tokens, two / four: 2,048 x 8,192 37.5 / 30.4, 2,048 x 2,048 11.9 / 10.5; 1 and 2 tokens,
// whose rings have three stages, 19.9 / 20.4 and 23.1 / 22.9: not; a tile on every SM leaves the next kernel's blocks no room
// beside, 2,368 x 4,096 12.2 / 13.0: not.  (Two more consumer warps, and the tokens' copies by a warp of
// their own, changed little: 23.1 and 20.6.)
constexpr int RT = 16, KC = 512, SL = KC / SLICE, LDR = KC + 4, LDX = SLICE + 4, ROW_THREADS = 96;

constexpr int rows_stage_floats(int mt) { return RT * LDR + mt * SL * LDX; }
constexpr int rows_stages(int mt, bool deep) { return deep ? (mt >= 8 ? 4 : 5) : (mt >= 4 ? 2 : 3); }
constexpr int rows_smem(int mt, bool deep) {
  return rows_stages(mt, deep) * rows_stage_floats(mt) * 4 + 2 * SL * RT * mt * 4 + 2 * rows_stages(mt, deep) * 8 + 16;
}

__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(s32(dst)), "l"(src), "r"(bytes), "r"(s32(bar)) : "memory");
}

template <int MT, bool DEEP>
__global__ void __launch_bounds__(ROW_THREADS)
sgemm_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                  long long lda, long long ldw, long long ldc, long long sa, long long sw, long long sc, int w_ahead, int* status) {
  constexpr int STAGES = rows_stages(MT, DEEP), SF = rows_stage_floats(MT);
  extern __shared__ __align__(128) float smem_f[];
  float* red = smem_f + STAGES * SF;                                  // [2][SL][RT][MT] slice values
  uint64_t* full = reinterpret_cast<uint64_t*>(red + 2 * SL * RT * MT);
  uint64_t* empty = full + STAGES;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + STAGES);
  A += (size_t)blockIdx.z * sa;
  W += (size_t)blockIdx.z * sw;
  C += (size_t)blockIdx.z * sc;
  bspec::pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 33);                        // the weights' byte count and every producer lane's tokens
      mbar_init(empty + s, 2);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // tiles: token chunks fastest, so that the blocks that need the same rows of W meet in the L2
  const int chunks = (M + MT - 1) / MT, tiles = (N + RT - 1) / RT * chunks, kcs = (K + KC - 1) / KC;
  if (warp == 2) {
    long long it = 0;
    auto weights = [&](int tile, int kc, int s) {
      const int n0 = tile / chunks * RT, k0 = kc * KC, len = min(KC, K - k0), rows = min(RT, N - n0);
      if (lane == 0) mbar_expect_tx(full + s, (uint32_t)rows * len * 4);
      __syncwarp();
      if (lane < rows) bulk_copy(smem_f + s * SF + lane * LDR, W + (size_t)(n0 + lane) * ldw + k0, len * 4, full + s);
    };
    auto tokens = [&](int tile, int kc, int s) {
      const int m0 = tile % chunks * MT, k0 = kc * KC, len = min(KC, K - k0), toks = min(MT, M - m0);
      for (int i = lane; i < MT * KC / 4; i += 32) {
        const int m = i / (KC / 4), c = i % (KC / 4) * 4;
        if (m < toks && c < len)
          copy_or_zero<true>(smem_f + s * SF + RT * LDR + (m * SL + c / SLICE) * LDX + c % SLICE, A + (size_t)(m0 + m) * lda + k0 + c, true);
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(s32(full + s)) : "memory");
    };
    // the first stages' weights need not wait for the kernel before this one, unless it may be writing them
    if (!w_ahead) bspec::pdl_wait();
    int pre = 0;
    for (int tile = blockIdx.x; tile < tiles && pre < STAGES; tile += gridDim.x)
      for (int kc = 0; kc < kcs && pre < STAGES; ++kc) weights(tile, kc, pre++);
    bspec::pdl_wait();
    bool ok = true;
    long long armed = 0;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x)
      for (int kc = 0; kc < kcs && ok; ++kc, ++it) {
        const int s = (int)(it % STAGES);
        if (it >= STAGES) {
          ok = mbar_wait(empty + s, (uint32_t)(it / STAGES - 1) & 1u, abort_flag, status, 91);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          weights(tile, kc, s);
        }
        tokens(tile, kc, s);
        armed = it + 1;
      }
    if (*abort_flag) {
      // let copies that are still in flight land before the block's shared memory is given up
      for (long long i = armed > STAGES ? armed - STAGES : 0; i < armed; ++i)
        for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(full + i % STAGES, (uint32_t)(i / STAGES) & 1u); ++t) __nanosleep(32);
    }
  } else {
    bspec::pdl_wait();                               // C may reuse memory that the kernel before still reads
    constexpr int OWN = (RT * MT + 63) / 64;         // output numbers whose slices this thread adds up
    const int r = tid % (RT / 2), sl = tid / (RT / 2);
    long long it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      float g[OWN], total[OWN];
      for (int kc = 0; kc < kcs; ++kc, ++it) {
        const int s = (int)(it % STAGES);
        ok = mbar_wait(full + s, (uint32_t)(it / STAGES) & 1u, abort_flag, status, 92);
        const int len = ok ? min(KC, K - kc * KC) - sl * SLICE : 0;
        const float* w_ = smem_f + s * SF + r * LDR + sl * SLICE;
        const float* x_ = smem_f + s * SF + RT * LDR + sl * LDX;
        float acc[MT][2][2];                          // [token][row][even, odd k]
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[m][0][0] = acc[m][0][1] = acc[m][1][0] = acc[m][1][1] = 0.f;
        const int quads = min(SLICE, max(len, 0)) / 4;
#pragma unroll 4
        for (int k = 0; k < quads; ++k) {
          const float4 w0 = *reinterpret_cast<const float4*>(w_ + 4 * k);
          const float4 w1 = *reinterpret_cast<const float4*>(w_ + RT / 2 * LDR + 4 * k);
#pragma unroll
          for (int m = 0; m < MT; ++m) {              // (scalar: packed multiply-adds were 7 % slower here)
            const float4 x = *reinterpret_cast<const float4*>(x_ + m * SL * LDX + 4 * k);
            acc[m][0][0] = fmaf(x.x, w0.x, acc[m][0][0]);
            acc[m][0][1] = fmaf(x.y, w0.y, acc[m][0][1]);
            acc[m][1][0] = fmaf(x.x, w1.x, acc[m][1][0]);
            acc[m][1][1] = fmaf(x.y, w1.y, acc[m][1][1]);
            acc[m][0][0] = fmaf(x.z, w0.z, acc[m][0][0]);
            acc[m][0][1] = fmaf(x.w, w0.w, acc[m][0][1]);
            acc[m][1][0] = fmaf(x.z, w1.z, acc[m][1][0]);
            acc[m][1][1] = fmaf(x.w, w1.w, acc[m][1][1]);
          }
        }
        float* red_ = red + (it & 1) * (SL * RT * MT);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          red_[(sl * RT + r) * MT + m] = acc[m][0][0] + acc[m][0][1];
          red_[(sl * RT + r + RT / 2) * MT + m] = acc[m][1][0] + acc[m][1][1];
        }
        ok = sync_and(ok);
        if (!ok) break;
        if (lane == 0) mbar_arrive(empty + s);
        const bool first = kc % (GROUP / KC) == 0, last = (kc + 1) % (GROUP / KC) == 0 || kc + 1 == kcs;
        const int slices = min(SL, (min(KC, K - kc * KC) + SLICE - 1) / SLICE);
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
          const int i = tid + 64 * o;
          if (i < RT * MT) {
            float v = first ? red_[i] : g[o] + red_[i];
            for (int q = 1; q < slices; ++q) v += red_[q * RT * MT + i];
            g[o] = v;
            if (last) total[o] = kc < GROUP / KC ? v : total[o] + v;
          }
        }
      }
      const int n0 = tile / chunks * RT, m0 = tile % chunks * MT;
      if (ok) {
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
          const int i = tid + 64 * o, n = n0 + i / MT, m = m0 + i % MT;
          if (i < RT * MT && n < N && m < M) C[(size_t)m * ldc + n] = total[o];
        }
      }
    }
  }
}

template <int MT, bool DEEP>
int launch_rows_ring(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                long long sa, long long sw, long long sc, int batch, int w_ahead, int* status, cudaStream_t stream) {
  static bool set[bspec::kMaxDevices] = {};
  bool& done = set[bspec::current_device()];
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(sgemm_rows_kernel<MT, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_smem(MT, DEEP));
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const int tiles = (N + RT - 1) / RT * ((M + MT - 1) / MT);
  const int fit = max(1, 2 * bspec::sm_count() / batch);
  BSPEC_LAUNCH((sgemm_rows_kernel<MT, DEEP>), dim3(min(tiles, fit), 1, batch), ROW_THREADS, rows_smem(MT, DEEP), stream, A, W, C, M, N, K, lda,
               ldw, ldc, sa, sw, sc, w_ahead, status);
  return BSPEC_LAUNCH_CHECK();
}

template <int MT>
int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                long long sa, long long sw, long long sc, int batch, int w_ahead, int* status, cudaStream_t stream) {
  if constexpr (MT >= 4)
    if ((long long)((N + RT - 1) / RT) * ((M + MT - 1) / MT) * batch < bspec::sm_count())
      return launch_rows_ring<MT, true>(A, W, C, M, N, K, lda, ldw, ldc, sa, sw, sc, batch, w_ahead, status, stream);
  return launch_rows_ring<MT, false>(A, W, C, M, N, K, lda, ldw, ldc, sa, sw, sc, batch, w_ahead, status, stream);
}

template <int BM, bool VEC>
int launch_tile(const float* A, const float* W, float* C, float* part, int M, int N, int K, long long lda, long long ldw,
                long long ldc, long long sa, long long sw, long long sc, int batch, int splits, cudaStream_t stream) {
  static bool set[bspec::kMaxDevices] = {};
  bool& done = set[bspec::current_device()];
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(sgemm_tile_kernel<BM, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<BM>::SMEM);
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const dim3 grid((N + Tile<BM>::BN - 1) / Tile<BM>::BN, (M + BM - 1) / BM, batch * splits);
  if (grid.y > 65535 || grid.z > 65535) return (int)cudaErrorInvalidConfiguration;
  BSPEC_LAUNCH((sgemm_tile_kernel<BM, VEC>), grid, Tile<BM>::NT, Tile<BM>::SMEM, stream, A, W, C, part, M, N, K, lda, ldw, ldc, sa, sw, sc,
               splits);
  return BSPEC_LAUNCH_CHECK();
}

constexpr int ROWS_MAX_M = 32;          // most rows of the kernel for few rows
constexpr long long SCRATCH_FLOATS = 64ll << 20;

// How many blocks along K the tile kernel takes: whole groups each, so that the last wave of blocks is well filled.
template <int BM>
int tile_splits(int M, int N, int K, int batch) {
  const int slots = bspec::sm_count() * Tile<BM>::PER_SM;
  const int groups = (K + GROUP - 1) / GROUP;
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + Tile<BM>::BN - 1) / Tile<BM>::BN) * batch;
  if (groups == 1 || tiles >= 4ll * slots || (long long)groups * M * N * batch > SCRATCH_FLOATS) return 1;
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= groups && (long long)s * batch <= 65535; ++s) {       // (batch x splits is a grid's z)
    const int per = (groups + s - 1) / s;
    const double waves = (double)((tiles * s + slots - 1) / slots);
    const double cost = waves * per + (s > 1 ? 0.25 : 0.0);          // the join: a pass over the groups' sums
    if (cost < best_cost - 1e-9) { best_cost = cost; best = s; }
  }
  return best;
}

struct TilePlan {
  int bm, splits;
};

// Rows of a tile and blocks along K.  Where the large tiles' blocks are fewer than the SMs, each of them works alone on its SM
// and a product takes the time of one: 32 x 32 tiles then.
TilePlan tile_plan(int M, int N, int K, int batch) {
  const int bm = M > 64 ? 128 : 64, splits = bm == 128 ? tile_splits<128>(M, N, K, batch) : tile_splits<64>(M, N, K, batch);
  const long long blocks = (long long)((M + bm - 1) / bm) * ((N + 63) / 64) * batch * splits;
  return blocks < bspec::sm_count() ? TilePlan{32, tile_splits<32>(M, N, K, batch)} : TilePlan{bm, splits};
}

bool rows_of_16_bytes(const float* A, const float* W, int K, long long lda, long long ldw, long long sa, long long sw) {
  return ((K | lda | ldw | sa | sw) & 3) == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
}
}  // namespace

// Floats of scratch that the product of these sizes wants (0: none).
BSPEC_API long long bspec_sgemm_scratch(const float* A, const float* W, int M, int N, int K, long long lda, long long ldw,
                                        long long sa, long long sw, int batch) {
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0 || (M <= ROWS_MAX_M && rows_of_16_bytes(A, W, K, lda, ldw, sa, sw))) return 0;
  return tile_plan(M, N, K, batch).splits > 1 ? (long long)((K + GROUP - 1) / GROUP) * M * N * batch : 0;
}

// `batch` products C_b = A_b * W_b^T whose operands lie sa / sw / sc elements apart.  ``scratch``: bspec_sgemm_scratch
// floats; ``w_ahead``: W is complete whatever still runs on the stream (a parameter), so it may be read before the kernel
// before this one ends; ``status``: the device's status word (0 unless a bounded wait ran out).
BSPEC_API int bspec_sgemm_tn_batched(const float* A, const float* W, float* C, int M, int N, int K, long long lda,
                                     long long ldw, long long ldc, long long sa, long long sw, long long sc, int batch,
                                     float* scratch, int w_ahead, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (batch > 65535) return (int)cudaErrorInvalidConfiguration;
  const bool vec = rows_of_16_bytes(A, W, K, lda, ldw, sa, sw);
  if (M <= ROWS_MAX_M && K > 0 && vec) {
    auto fn = M == 1 ? launch_rows<1> : (M == 2 ? launch_rows<2> : (M <= 4 ? launch_rows<4> : launch_rows<8>));
    return fn(A, W, C, M, N, K, lda, ldw, ldc, sa, sw, sc, batch, w_ahead, status, stream);
  }
  const TilePlan plan = tile_plan(M, N, K, batch);
  const int groups = (K + GROUP - 1) / GROUP, splits = K > 0 && scratch != nullptr ? plan.splits : 1;
  auto fn = plan.bm == 128 ? (vec ? launch_tile<128, true> : launch_tile<128, false>)
            : (plan.bm == 64 ? (vec ? launch_tile<64, true> : launch_tile<64, false>) : (vec ? launch_tile<32, true> : launch_tile<32, false>));
  const int err = fn(A, W, C, scratch, M, N, K, lda, ldw, ldc, sa, sw, sc, batch, splits, stream);
  if (err != 0 || splits == 1) return err;
  const long long blocks = ((long long)M * N + 255) / 256;
  BSPEC_LAUNCH((sgemm_join_kernel), dim3((unsigned)min(blocks, 8ll * bspec::sm_count()), batch), 256, 0, stream, scratch, C, M, N,
               ldc, sc, groups);
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_DEFINE_TRACE_SETTER(bspec_trace_set_gemm_fp32)
