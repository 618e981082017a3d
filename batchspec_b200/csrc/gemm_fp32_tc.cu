// float32 matrix product on the tensor cores, for operands with many rows:  C[M,N] = A[M,K] * W[N,K]^T, all row-major.
//
// A float32 number is the sum of three bfloat16 numbers (8 significant bits each, rounded to nearest, every remainder
// exact): x = x1 + x2 + x3.  Of the nine products of two such sums the six of at most 2^-16 of the whole are formed,
// x1 y1 + (x1 y2 + x2 y1) + (x1 y3 + x2 y2 + x3 y1); each is exact in float32, and what is left out is below 2^-25 of
// |x y|.  (The tensor core takes parts below the smallest normal number, 2^-126, as zero: numbers below 2^-102 lose digits.)  The tensor core's accumulator rounds towards zero, so it never carries a long sum: it takes SPAN numbers of K,
// smallest products first, and what it has then is added in float32, rounded to nearest, by the threads that read it:
//   span    32 k in the tensor core;
//   group   512 k: its spans, added in order;
//   result  the groups, added in order.
// The order depends on K alone: a row's bits depend neither on M nor on how the work is cut.
// Relative error against 64 bits (2-norm, normal operands): 1.04e-7 at K = 2,048 and 1.23e-7 at 8,192, where the chains of
// multiply-adds of gemm_fp32.cu have 1.34e-7 and 1.43e-7; with spans of 64 k 3.2e-7, of 128 k 7.5e-7.
//
//   split_kernel  A -> three bfloat16 planes [3][M][K rounded up to 64], zeros past K;
//   sgemm_tc_kernel  one persistent CTA per SM, tiles of 128 rows of W x 128 rows of A, 16 warps:
//     warp 0   TMA: A's planes, 64 k of 128 rows at a time, three stages of 48 KB;
//     warp 2   TMA: W as it is, float32, 32 k of 128 rows at a time, four stages of 16 KB;
//     warps 4-7   one thread per row of W: takes a stage's 32 numbers apart and leaves them in tensor memory, the A
//              operand of the products (four stages of 48 columns).  W is never written anywhere as three planes;
//     warp 1   one thread issues the 12 tcgen05.mma of a span (128 x 128 x 16, A from tensor memory, B from shared memory);
//     warps 8-15   one thread per row of W and 64 columns: add the spans (two accumulators of 128 columns alternate).
// On a B200, against the packed multiply-adds of gemm_fp32.cu: 967 x 16,384 x 2,048 1,684 -> 488 us, 967 x 2,048 x 2,048
// 258 -> 83, 967 x 2,048 x 8,192 863 -> 335.
#include "tma.cuh"
#include "umma.cuh"
#include <float.h>

using namespace bspec;

namespace {

constexpr int TN = 128;                            // rows of W = accumulator rows
constexpr int TT = 128;                            // rows of A = accumulator columns
constexpr int KB = 64, SPAN = 32, GROUP = 512;
constexpr int MIN_ROWS = 192;
constexpr double MIN_WORK = 1 << 28;
constexpr int B_STAGES = 3, W_STAGES = 4, A_STAGES = 4;
constexpr int PLANE = TT * KB * 2;                 // bytes of one plane of a stage
constexpr int B_BYTES = 3 * PLANE, W_BYTES = TN * SPAN * 4;
constexpr int THREADS = 512;
constexpr int A_COL = 2 * TT, A_COLS = 48;         // tensor memory: two accumulators, then the stages of W's planes
constexpr int SMEM = 1024 + B_STAGES * B_BYTES + W_STAGES * W_BYTES + 256;
// registers per thread of the four warpgroups once the roles are taken: their sum is at most four times what the kernel
// is launched with (128: 512 threads)
constexpr int REGS_IO = 40, REGS_SPLIT = 72, REGS_ADD = 200;
static_assert(REGS_IO + REGS_SPLIT + 2 * REGS_ADD <= 4 * 128, "more registers than the block has");
static_assert(A_COL + A_STAGES * A_COLS <= 512, "tensor memory");

__device__ __forceinline__ void load_box3(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(s32(dst)), "l"(map), "r"(s32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
// two numbers as three pairs of bfloat16 numbers (the first in the low half)
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  auto pair = [](float a, float b) -> uint32_t {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  p1 = pair(x0, x1);
  x0 -= __uint_as_float(p1 << 16);
  x1 -= __uint_as_float(p1 & 0xffff0000u);
  p2 = pair(x0, x1);
  x0 -= __uint_as_float(p2 << 16);
  x1 -= __uint_as_float(p2 & 0xffff0000u);
  p3 = pair(x0, x1);
}

// ------------------------------------------------------------------------------------------------ A into planes
// A thread takes four numbers of a row.  Bound by memory: 4 bytes in, 6 out per number.
template <bool VEC>
__global__ void __launch_bounds__(256)
split_kernel(const float* __restrict__ A, uint2* __restrict__ planes, int M, int K, long long lda, int Kp) {
  bspec::pdl_prologue(10);
  const int quads = Kp / 4;
  const long long total = (long long)M * quads;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const int m = (int)(i / quads), k = (int)(i - (long long)m * quads) * 4;
    const float* src = A + (size_t)m * lda + k;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (VEC && k + 4 <= K) {
      const float4 f = *reinterpret_cast<const float4*>(src);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k + j < K) v[j] = src[j];
    }
    uint2 p[3];
    split2(v[0], v[1], p[0].x, p[1].x, p[2].x);
    split2(v[2], v[3], p[0].y, p[1].y, p[2].y);
#pragma unroll
    for (int j = 0; j < 3; ++j) planes[j * total + i] = p[j];
  }
}

struct Params {
  const float* A;
  const float* W;
  float* C;
  float* part;               // [groups][M][N] when the groups of a tile are dealt to several CTAs, else null
  int* status;
  int M, N, K;
  long long lda, ldw, ldc;
  int splits, per;           // CTAs along K, groups of each
};

// The sum over k_begin .. k_end of one output on the CUDA cores, for results that are not finite: an infinity is no sum
// of three bfloat16 numbers that products could be formed of.
__device__ __forceinline__ float plain_sum(const float* __restrict__ a, const float* __restrict__ w, int k_begin, int k_end) {
  float total = 0.f;
  for (int k0 = k_begin; k0 < k_end; k0 += 64) {
    float even = 0.f, odd = 0.f;
    for (int k = k0; k < min(k0 + 64, k_end); k += 2) {
      even = fmaf(a[k], w[k], even);
      if (k + 1 < k_end) odd = fmaf(a[k + 1], w[k + 1], odd);
    }
    total += even + odd;
  }
  return total;
}

__global__ void __launch_bounds__(THREADS, 1)
sgemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char* b_ring = smem;
  unsigned char* w_ring = smem + B_STAGES * B_BYTES;
  uint64_t* b_full = reinterpret_cast<uint64_t*>(w_ring + W_STAGES * W_BYTES);
  uint64_t* b_empty = b_full + B_STAGES;
  uint64_t* w_full = b_empty + B_STAGES;
  uint64_t* w_empty = w_full + W_STAGES;
  uint64_t* a_full = w_empty + W_STAGES;
  uint64_t* a_empty = a_full + A_STAGES;
  uint64_t* d_full = a_empty + A_STAGES;
  uint64_t* d_empty = d_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(d_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < B_STAGES; ++s) { mbar_init(b_full + s, 1); mbar_init(b_empty + s, 1); }
    for (int s = 0; s < W_STAGES; ++s) { mbar_init(w_full + s, 1); mbar_init(w_empty + s, 4); }
    for (int s = 0; s < A_STAGES; ++s) { mbar_init(a_full + s, 4); mbar_init(a_empty + s, 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(d_full + s, 1); mbar_init(d_empty + s, 8); }
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

  // Items: tiles with the tiles of A fastest (CTAs that start together share W in the L2), slices of K slowest.
  const int mt = (p.M + TT - 1) / TT, nt = (p.N + TN - 1) / TN, blocks = (p.K + KB - 1) / KB;
  const int tiles = mt * nt, items = tiles * p.splits;
  auto block_range = [&](int item, int& kb0, int& kb1) {
    const int split = item / tiles;
    kb0 = min(blocks, split * p.per * (GROUP / KB));
    kb1 = min(blocks, kb0 + p.per * (GROUP / KB));
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_IO));
    if (warp == 0 && lane == 0) {
      // ------------------------------------------------------------------ A's planes
      uint32_t n = 0, armed = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int kb0, kb1;
        block_range(item, kb0, kb1);
        const int m0 = item % tiles % mt * TT;
        for (int kb = kb0; kb < kb1 && ok; ++kb, ++n) {
          const uint32_t s = n % B_STAGES;
          ok = mbar_wait(b_empty + s, ((n / B_STAGES) & 1u) ^ 1u, abort_flag, p.status, 95);
          if (!ok) break;
          mbar_expect_tx(b_full + s, B_BYTES);
          load_box3(b_ring + s * B_BYTES, &map_x, b_full + s, kb * KB, m0, 0);
          armed = n + 1;
        }
      }
      if (*abort_flag)           // copies still in flight land before the block's shared memory is given up
        for (uint32_t i = armed > B_STAGES ? armed - B_STAGES : 0; i < armed; ++i)
          for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(b_full + i % B_STAGES, (i / B_STAGES) & 1u); ++t) __nanosleep(32);
    } else if (warp == 2 && lane == 0) {
      // ------------------------------------------------------------------ W
      uint32_t n = 0, armed = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int kb0, kb1;
        block_range(item, kb0, kb1);
        const int n0 = item % tiles / mt * TN;
        for (int c = 2 * kb0; c < 2 * kb1 && ok; ++c, ++n) {
          const uint32_t s = n % W_STAGES;
          ok = mbar_wait(w_empty + s, ((n / W_STAGES) & 1u) ^ 1u, abort_flag, p.status, 96);
          if (!ok) break;
          mbar_expect_tx(w_full + s, W_BYTES);
          tma_load_2d(w_ring + s * W_BYTES, &map_w, w_full + s, c * SPAN, n0);
          armed = n + 1;
        }
      }
      if (*abort_flag)
        for (uint32_t i = armed > W_STAGES ? armed - W_STAGES : 0; i < armed; ++i)
          for (uint32_t t = 0; t < (1u << 16) && !mbar_try_wait(w_full + i % W_STAGES, (i / W_STAGES) & 1u); ++t) __nanosleep(32);
    } else if (warp == 1 && lane == 0) {
      // ------------------------------------------------------------------ the products of a span, smallest first
      const uint32_t idesc = instr_desc(TT);
      uint32_t nb = 0, na = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int kb0, kb1;
        block_range(item, kb0, kb1);
        for (int kb = kb0; kb < kb1 && ok; ++kb, ++nb) {
          const uint32_t bs = nb % B_STAGES;
          ok = mbar_wait(b_full + bs, (nb / B_STAGES) & 1u, abort_flag, p.status, 97);
          if (!ok) break;
          const uint64_t bdesc = smem_desc(b_ring + bs * B_BYTES);
          for (int h = 0; h < 2 && ok; ++h, ++na) {
            const uint32_t as = na % A_STAGES, db = na & 1u;
            ok = mbar_wait(d_empty + db, ((na >> 1) & 1u) ^ 1u, abort_flag, p.status, 98);
            if (ok) ok = mbar_wait(a_full + as, (na / A_STAGES) & 1u, abort_flag, p.status, 99);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem + db * TT, a = tmem + A_COL + as * A_COLS;
            constexpr int PW[6] = {2, 1, 0, 1, 0, 0}, PX[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
            for (int q = 0; q < 6; ++q)
#pragma unroll
              for (int s = 0; s < 2; ++s)
                tc_mma_a_tmem(d, a + PW[q] * 16 + s * 8, bdesc + (uint64_t)(PX[q] * (PLANE >> 4) + (2 * h + s) * 2), idesc,
                              (q > 0 || s > 0) ? 1u : 0u);
            tc_commit(a_empty + as);
            tc_commit(d_full + db);
          }
          if (ok) tc_commit(b_empty + bs);
        }
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ W into planes in tensor memory, a thread per row
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_SPLIT));
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t n = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      int kb0, kb1;
      block_range(item, kb0, kb1);
      for (int c = 2 * kb0; c < 2 * kb1; ++c, ++n) {
        const uint32_t ws = n % W_STAGES, as = n % A_STAGES;
        ok = mbar_wait(w_full + ws, (n / W_STAGES) & 1u, abort_flag, p.status, 100);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        uint32_t p1[16], p2[16], p3[16];
        const unsigned char* src = w_ring + ws * W_BYTES + row * 128;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 f = *reinterpret_cast<const float4*>(src + ((q ^ (row & 7)) << 4));
          split2(f.x, f.y, p1[2 * q], p2[2 * q], p3[2 * q]);
          split2(f.z, f.w, p1[2 * q + 1], p2[2 * q + 1], p3[2 * q + 1]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(w_empty + ws);
        ok = mbar_wait(a_empty + as, ((n / A_STAGES) & 1u) ^ 1u, abort_flag, p.status, 101);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t dst = tmem + A_COL + as * A_COLS + lane_addr;
        tc_st16(dst, p1);
        tc_st16(dst + 16, p2);
        tc_st16(dst + 32, p3);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full + as);
      }
    }
  } else {
    // ------------------------------------------------------------------ the spans' sums
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_ADD));
    const int half = (warp - 8) >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t src0 = tmem + ((uint32_t)((warp & 3) * 32) << 16) + half * 64;
    uint32_t nd = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      int kb0, kb1;
      block_range(item, kb0, kb1);
      const int tile = item % tiles, m0 = tile % mt * TT + half * 64, n = tile / mt * TN + row;
      uint64_t acc[32], total[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = total[j] = 0ull;
      auto store = [&](uint64_t (&v)[32], float* out, long long ld, int k_begin, int k_end) {
        if (n >= p.N) return;
        out += (size_t)m0 * ld + n;
        const int rows = min(64, p.M - m0);
        bool finite = true;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const float x = __uint_as_float((uint32_t)(j & 1 ? v[j >> 1] >> 32 : v[j >> 1]));
          if (j < rows) {
            out[(size_t)j * ld] = x;
            finite = finite && fabsf(x) <= FLT_MAX;
          }
        }
        if (!finite)
          for (int j = 0; j < rows; ++j)
            if (!(fabsf(out[(size_t)j * ld]) <= FLT_MAX))
              out[(size_t)j * ld] = plain_sum(p.A + (size_t)(m0 + j) * p.lda, p.W + (size_t)n * p.ldw, k_begin, k_end);
      };
      const int c_end = 2 * kb1;
      for (int c = 2 * kb0; c < c_end; ++c, ++nd) {
        const uint32_t db = nd & 1u;
        ok = mbar_wait(d_full + db, (nd >> 1) & 1u, abort_flag, p.status, 102);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        constexpr int PER_GROUP = GROUP / SPAN;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t v[16];
          tc_ld16(src0 + db * TT + 16 * q, v);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc[8 * q + j] = add2(acc[8 * q + j], pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(d_empty + db);
        if (c % PER_GROUP == PER_GROUP - 1 || c + 1 == c_end) {
          const int g = c / PER_GROUP;
          if (p.part != nullptr) {
            store(acc, p.part + (size_t)g * p.M * p.N, p.N, g * GROUP, min(p.K, (g + 1) * GROUP));
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) total[j] = add2(total[j], acc[j]);
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[j] = 0ull;
        }
      }
      if (ok && p.part == nullptr) store(total, p.C, p.ldc, 0, p.K);
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

// C = the groups' sums, added in order
__global__ void __launch_bounds__(256)
join_groups_kernel(const float* __restrict__ part, float* __restrict__ C, long long mn, int groups) {
  bspec::pdl_prologue(10);
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < mn / 4; i += (long long)gridDim.x * 256) {
    float4 v = *reinterpret_cast<const float4*>(part + 4 * i);
    for (int g = 1; g < groups; ++g) {
      const float4 o = *reinterpret_cast<const float4*>(part + g * mn + 4 * i);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    *reinterpret_cast<float4*>(C + 4 * i) = v;
  }
}

long long plane_bytes(int M, int K) { return (3ll * M * ((K + KB - 1) / KB * KB) * 2 + 255) / 256 * 256; }

// CTAs along K: whole groups each, so that the last wave of CTAs is well filled.  In units of a group's time in a CTA, about
// 16 us; the groups' sums, written and read again at some 5 TB/s, are what it costs (967 x 2,048 x 8,192, 128 tiles of 16 groups:
// sliced: 336 us, whole: 279).
int tc_splits(int M, int N, int K) {
  const long long tiles = (long long)((M + TT - 1) / TT) * ((N + TN - 1) / TN);
  const int groups = (K + GROUP - 1) / GROUP;
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= groups; ++s) {
    const int per = (groups + s - 1) / s;
    const long long waves = (tiles * s + bspec::sm_count() - 1) / bspec::sm_count();
    const double cost = (double)waves * per + (s > 1 ? 0.3 + 8.0 * groups * M * N / 80e6 : 0.0);
    if (cost < best_cost - 1e-9) { best_cost = cost; best = s; }
  }
  return best;
}

// Which products come here.  From 33 rows on this kernel is the faster one (33 x 16,384 x 2,048 79 against 136 us); up to
// 191 rows the chains of gemm_fp32.cu stay, so that a decode step, a short prompt and a portion give a row the same bits.
// Small products do not pay for the taking apart and the pipeline's filling, us, multiply-adds / here: 512 x 512 x 512 20.5 / 28.5,
// 2,048 x 256 x 256 18.5 / 21.5; 2^28 and more: 1,024 x 512 x 512 28.8 / 28.7, 256 x 512 x 2,048 33.8 / 32.7, 1,024^3 78 / 36,
// 4,096 x 128 x 2,048 90 / 48, 192 x 2,048 x 2,048 71 / 35.
bool takes(const float* W, int M, int N, int K, long long ldw) {
  return M >= MIN_ROWS && N % 4 == 0 && K >= SPAN && (ldw & 3) == 0 && ((uintptr_t)W & 15) == 0 &&
         (double)M * N * K >= MIN_WORK;
}
}  // namespace

// Bytes of scratch (0: the product of these sizes is not for this kernel).
BSPEC_API long long bspec_sgemm_tc_scratch(const float* W, int M, int N, int K, long long ldw) {
  if (!takes(W, M, N, K, ldw)) return 0;
  return plane_bytes(M, K) + (tc_splits(M, N, K) > 1 ? (long long)((K + GROUP - 1) / GROUP) * M * N * 4 : 0);
}
// Kernels that it launches.
BSPEC_API int bspec_sgemm_tc_launches(int M, int N, int K) { return tc_splits(M, N, K) > 1 ? 3 : 2; }

BSPEC_API int bspec_sgemm_tc(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw,
                             void* scratch, int* status, cudaStream_t stream) {
  if (!takes(W, M, N, K, ldw)) return (int)cudaErrorInvalidValue;
  const int Kp = (K + KB - 1) / KB * KB, splits = tc_splits(M, N, K), groups = (K + GROUP - 1) / GROUP;
  static bool set[bspec::kMaxDevices] = {};
  bool& done = set[bspec::current_device()];
  if (!done) {
    cudaFuncAttributes at;
    cudaError_t e = cudaFuncGetAttributes(&at, sgemm_tc_kernel);
    if (e != cudaSuccess) return (int)e;
    if (at.numRegs < 128) return (int)cudaErrorInvalidConfiguration;      // the roles' registers would not fit the block's
    e = cudaFuncSetAttribute(sgemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  auto fn = encode_fn();
  if (fn == nullptr) return (int)cudaErrorInvalidValue;
  CUtensorMap map_w, map_x;
  {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, strides[1] = {(cuuint64_t)ldw * 4};
    cuuint32_t box[2] = {SPAN, TN}, elem[2] = {1, 1};
    if (fn(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return (int)cudaErrorInvalidValue;
  }
  {
    cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)M, 3}, strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)M * Kp * 2};
    cuuint32_t box[3] = {KB, TT, 3}, elem[3] = {1, 1, 1};
    if (fn(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, scratch, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return (int)cudaErrorInvalidValue;
  }
  const long long quads = (long long)M * (Kp / 4);
  const unsigned sb = (unsigned)min((quads + 255) / 256, (long long)bspec::sm_count() * 16);
  const bool vec = (lda & 3) == 0 && ((uintptr_t)A & 15) == 0;
  if (vec) BSPEC_LAUNCH((split_kernel<true>), sb, 256, 0, stream, A, (uint2*)scratch, M, K, lda, Kp);
  else BSPEC_LAUNCH((split_kernel<false>), sb, 256, 0, stream, A, (uint2*)scratch, M, K, lda, Kp);
  Params p;
  p.A = A; p.W = W; p.C = C;
  p.part = splits > 1 ? reinterpret_cast<float*>((char*)scratch + plane_bytes(M, K)) : nullptr;
  p.status = status;
  p.M = M; p.N = N; p.K = K;
  p.lda = lda; p.ldw = ldw; p.ldc = N;
  p.splits = splits;
  p.per = (groups + splits - 1) / splits;
  const long long items = (long long)((M + TT - 1) / TT) * ((N + TN - 1) / TN) * splits;
  if (items > (1ll << 30)) return (int)cudaErrorInvalidConfiguration;
  BSPEC_LAUNCH(sgemm_tc_kernel, dim3((unsigned)min(items, (long long)bspec::sm_count())), THREADS, SMEM, stream, map_w, map_x, p);
  int err = BSPEC_LAUNCH_CHECK();
  if (err != 0 || splits == 1) return err;
  const long long mn = (long long)M * N;
  BSPEC_LAUNCH(join_groups_kernel, dim3((unsigned)min((mn / 4 + 255) / 256, 8ll * bspec::sm_count())), 256, 0, stream,
               (const float*)p.part, C, mn, groups);
  return BSPEC_LAUNCH_CHECK();
}

BSPEC_DEFINE_TRACE_SETTER(bspec_trace_set_gemm_fp32_tc)
