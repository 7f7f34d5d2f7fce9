// Linear layer of float32 rows on the 5th-generation tensor cores, at float32's precision:
//   C[M,N] = epilogue(A[M,K] . W[N,K]^T + bias[N]) (+ residual[M,N]),  all of them float32
//
// Every operand is the sum of three bfloat16 numbers, x = h + m + l (24 bits together, nothing of x is lost down to 2^-110, below which
// l, and then m, ends with bfloat16's range; h is cut off, m rounded, so that l has either sign), and a product of two operands is
// the six products of such parts that reach 24 bits: h h, h m, m h, h l, l h, m m.  What is left out, m l, l m and l l, is up to 2^-22 of
// the product where both mantissas are at their worst, 2^-25.4 in the mean square, and as often above as below: less than the rounding
// of a running sum by each FMA.  The tensor core's products are exact; what
// it adds to its accumulator it cuts off instead of rounding, so no sum is left to it for long: a block of 64 of K starts a
// fresh accumulator, the five small products of all its steps go in first, when the accumulator is 2^-8 of what it will be,
// the four steps of h h last, and the block's sum is added, rounded to nearest, to a sum in registers.  One order for every
// tile width and number of rows, so a row's result does not depend on how many other rows go through this kernel; it differs by rounding
// from the FMA kernels', and which of them a row takes depends on its own request alone (parts/linear.py).
//
// 737 rows, weights from DRAM: 3072 x 1024 35 us, 1024 x 1024 24, 4096 x 1024 64, 1024 x 4096 79 (FMA tiles: 144, 73, 212, 278); eight
// warps taking the numbers apart instead of sixteen: 43, 30, 76, 98 (they wait for what they read most of the time).
// What bounds it is reading the operands and taking them apart: 4096 x 1024 issues instructions in 70 % of all cycles, its tensor pipes
// are busy in 25 %, shared memory in 30 %.
//
// Per CTA, over 128 x BN tiles (persistent, BN = 128 or 64):
//   warps 0-15   read the next block of A and W with 16-byte loads (registers hold a block while the one before is at work),
//                take it apart and store the six planes, 128-byte swizzled, into one of two buffers
//   warp 24      issues the 24 products of a block, commits the buffer back and the accumulator forward (two of them)
//   warps 16-23  add the accumulator of every block to their sums (64 columns of a row each at BN = 128); after the last
//                block bias, activation and residual, and out through shared memory as whole sectors
// Outputs that are not finite are computed again by their warp with plain FMAs, after all others of its tile: parts of an infinity, or
// sums beyond float32's range on the way, say nothing.  One row of NaN among 737 takes 4096 x 1024 from 63 to 80 us, all rows to 1.7 ms.
//
// Every wait on an mbarrier is bounded (tcgen05.cuh): after the limit all roles leave their loops, the CTA waits, bounded, for the
// products in flight, reports MLXB_ST_WAIT_TIMEOUT, frees its tensor memory and returns.
//
// K and the row strides are multiples of 4 elements, base addresses 16-byte aligned.
#include "activations.cuh"
#include "tcgen05.cuh"

MLXB_DEFINE_LAST_ERROR()

constexpr int BM = 128, BK = 64;
constexpr int SPLIT_WARPS = 16, SUM_WARPS = 8, MMA_WARP = SPLIT_WARPS + SUM_WARPS;
// whole groups of four warps, which registers are handed out to: 4 x 64 + 2 x 96 + 48 of the 7 x 72 of the launch
constexpr int THREADS = 32 * (MMA_WARP + 4);
constexpr int SPLIT_REGS = 64, SUM_REGS = 96, MMA_REGS = 48;
static_assert(SPLIT_WARPS * SPLIT_REGS + SUM_WARPS * SUM_REGS + 4 * MMA_REGS <= 28 * 72, "a larger sum would wait forever");
template <int R>
__device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

template <int BN>
struct Smem {
  alignas(1024) __nv_bfloat16 a[2][3][BM * BK];      // [buffer][part]
  alignas(1024) __nv_bfloat16 w[2][3][BN * BK];
  alignas(16) uint4 stage[SUM_WARPS][32 * 4];        // 64 bytes of each of a warp's 32 rows on their way out
  uint32_t bad[SUM_WARPS][BN / 8];                   // per eight rows and 16 columns the pieces of four columns that are not finite
  uint64_t full[2], empty[2];                        // a buffer's parts are written / have been multiplied
  uint64_t acc_full[2], acc_empty[2];
  uint64_t drained;                                  // abort path only
  uint32_t tmem_base;
  int abort_flag;
};

// Four neighbours taken apart, into the three planes at byte offset `at`: h is the number's upper half as it stands, m the nearest to
// what that leaves (16 bits), and what is left then (8 bits) is a bfloat16 number as it stands: one conversion for two numbers,
// and conversions run at an eighth of the rate of other instructions.
__device__ __forceinline__ uint32_t upper_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }
__device__ __forceinline__ void put_parts(const float4& v, char* plane0, uint32_t plane_bytes, uint32_t at) {
  const float x[4] = {v.x, v.y, v.z, v.w};
  uint32_t u[4], h[2], m[2], l[2];
  float r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    u[i] = __float_as_uint(x[i]);
    r[i] = x[i] - __uint_as_float(u[i] & 0xffff0000u);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    h[i] = upper_halves(u[2 * i], u[2 * i + 1]);
    const __nv_bfloat162 c = __floats2bfloat162_rn(r[2 * i], r[2 * i + 1]);
    m[i] = *reinterpret_cast<const uint32_t*>(&c);
    r[2 * i] -= __uint_as_float(m[i] << 16);
    r[2 * i + 1] -= __uint_as_float(m[i] & 0xffff0000u);
    l[i] = upper_halves(__float_as_uint(r[2 * i]), __float_as_uint(r[2 * i + 1]));
  }
  *reinterpret_cast<uint2*>(plane0 + at) = make_uint2(h[0], h[1]);
  *reinterpret_cast<uint2*>(plane0 + plane_bytes + at) = make_uint2(m[0], m[1]);
  *reinterpret_cast<uint2*>(plane0 + 2 * plane_bytes + at) = make_uint2(l[0], l[1]);
}

// 16 columns of a row's accumulator and the wait for them in one statement: between two the compiler may put additions of
// registers that the load has not written yet.
__device__ __forceinline__ void tmem_get16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}

// A row of A times up to four neighbouring rows of W in plain float32, by a warp; the same in every lane.
__device__ __noinline__ float4 plain_dots(const float* a, const float* w, int rows, int K) {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
  for (int k = (threadIdx.x & 31) * 4; k < K; k += 128) {
    const float4 x = *reinterpret_cast<const float4*>(a + k);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e >= rows) continue;
      const float4 y = *reinterpret_cast<const float4*>(w + (size_t)e * K + k);
      s[e] = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s[e]))));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
  return make_float4(s[0], s[1], s[2], s[3]);
}

__device__ __forceinline__ int stage_index(int row, int piece) { return row * 4 + (piece ^ ((row >> 1) & 3)); }

template <int BN, int EPI>
__global__ void __launch_bounds__(THREADS, 1)
linear_split_kernel(const float* A, const float* __restrict__ W, const float* __restrict__ bias, const float* residual, float* C,
                    int M, int N, int K, int lda, int ldc, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  Smem<BN>& sm = *reinterpret_cast<Smem<BN>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blocks = (K + BK - 1) / BK;
  const int tiles_m = (M + BM - 1) / BM, n_tiles = tiles_m * ((N + BN - 1) / BN);
  auto tile_m0 = [&](int t) { return (t % tiles_m) * BM; };
  auto tile_n0 = [&](int t) { return (t / tiles_m) * BN; };
  constexpr uint32_t TMEM_COLS = 2 * BN;

  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.full[b], SPLIT_WARPS);
      mbar_init(&sm.empty[b], 1);
      mbar_init(&sm.acc_full[b], 1);
      mbar_init(&sm.acc_empty[b], SUM_WARPS);
    }
    mbar_init(&sm.drained, 1);
    sm.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  volatile int* abort_flag = &sm.abort_flag;
  pdl_trigger();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = sm.tmem_base;

  if (warp < SPLIT_WARPS) {
    fewer_registers<SPLIT_REGS>();
    // 16 threads take the 64 k of a row, four each: a thread has rows tr, tr + ROWS, ... of A and of W
    constexpr int ROWS = 2 * SPLIT_WARPS, AR = BM / ROWS, WR = BN / ROWS;
    const int tr = threadIdx.x >> 4, tk = (threadIdx.x & 15) * 4;
    float4 av[AR], wv[WR];
    int tile = blockIdx.x, kb = 0;                     // the block that is asked for next
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch_w = [&]() {
      const int n0 = tile_n0(tile) + tr, k = kb * BK + tk;
      const bool in = tile < n_tiles && k < K;
      const float* p = W + (size_t)n0 * K + k;
#pragma unroll
      for (int i = 0; i < WR; ++i) wv[i] = in && n0 + ROWS * i < N ? *reinterpret_cast<const float4*>(p + (size_t)(ROWS * i) * K) : zero;
    };
    auto fetch_a = [&]() {
      const int m0 = tile_m0(tile) + tr, k = kb * BK + tk;
      const bool in = tile < n_tiles && k < K;
      const float* p = A + (size_t)m0 * lda + k;
#pragma unroll
      for (int i = 0; i < AR; ++i) av[i] = in && m0 + ROWS * i < M ? *reinterpret_cast<const float4*>(p + (size_t)(ROWS * i) * lda) : zero;
    };
    fetch_w();
    pdl_wait();                                        // A (and the residual) come from the kernel before
    A = after_wait(A);
    fetch_a();
    // rows ROWS apart have the same place in their group of eight: one swizzle for all of a thread's pieces
    const uint32_t at = (uint32_t)tr * 128 + (((uint32_t)(tk >> 3) ^ (tr & 7)) << 4) + (tk & 4) * 2;
    int it = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
      int kt = 0;
      for (; kt < blocks; ++kt, ++it) {
        const int b = it & 1;
        if (!mbar_wait_warp(&sm.empty[b], ((it >> 1) & 1) ^ 1, abort_flag)) break;
        char* pa = reinterpret_cast<char*>(sm.a[b][0]);
        char* pw = reinterpret_cast<char*>(sm.w[b][0]);
        if (++kb == blocks) { kb = 0; tile += gridDim.x; }
        // one operand's next block is on its way while the other's is taken apart
#pragma unroll
        for (int i = 0; i < WR; ++i) put_parts(wv[i], pw, BN * BK * 2, at + i * ROWS * 128);
        fetch_w();
#pragma unroll
        for (int i = 0; i < AR; ++i) put_parts(av[i], pa, BM * BK * 2, at + i * ROWS * 128);
        fetch_a();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.full[b]);
      }
      if (kt < blocks) break;
    }
  } else if (warp >= MMA_WARP) {
    fewer_registers<MMA_REGS>();
    constexpr uint32_t idesc = umma_idesc(BM, BN);
    constexpr uint32_t A_PART = BM * BK * 2 / 16, W_PART = BN * BK * 2 / 16;      // in units of 16 bytes
    const uint64_t da0 = umma_desc(smem_u32(sm.a[0][0])), dw0 = umma_desc(smem_u32(sm.w[0][0]));
    int it = 0;
    bool ok = warp == MMA_WARP;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x)
      for (int kt = 0; kt < blocks; ++kt, ++it) {
        const int b = it & 1;
        ok = mbar_wait_warp(&sm.acc_empty[b], ((it >> 1) & 1) ^ 1, abort_flag) &&
             mbar_wait_warp(&sm.full[b], (it >> 1) & 1, abort_flag);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_base + (uint32_t)(b * BN);
        const uint64_t da = da0 + (uint32_t)(b * 3) * A_PART, dw = dw0 + (uint32_t)(b * 3) * W_PART;
        if (elect_one()) {
          // (part of A, part of W), the smallest products first
          constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
          for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_bf16(acc, da + PA[p] * A_PART + 2 * k, dw + PW[p] * W_PART + 2 * k, idesc, p + k > 0 ? 1u : 0u);
          umma_commit(&sm.empty[b]);
#ifdef MLXB_TEST_WAIT_TIMEOUT
          if (!g_test_withhold_arrival || it > 0)      // the test's missing arrival
#endif
          umma_commit(&sm.acc_full[b]);
        }
        __syncwarp();
      }
  } else {
    more_registers<SUM_REGS>();
    // warp w may touch lanes 32 (w % 4) .. of tensor memory; the two warps of a quadrant share the tile's columns
    const int q = warp & 3, half = (warp - SPLIT_WARPS) >> 2;
    constexpr int COLS = BN / 2;
    pdl_wait();
    A = after_wait(A);
    residual = after_wait(residual);
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * COLS);
    uint4* stg = sm.stage[warp - SPLIT_WARPS];
    const int o_row = lane >> 2, o_piece = lane & 3;
    int it = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
      float sum[COLS];
#pragma unroll
      for (int i = 0; i < COLS; ++i) sum[i] = 0.f;
      int kt = 0;
      for (; kt < blocks; ++kt, ++it) {
        const int b = it & 1;
        if (!mbar_wait_warp(&sm.acc_full[b], (it >> 1) & 1, abort_flag)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < COLS; c += 16) {
          uint32_t r[16];
          tmem_get16(taddr + (uint32_t)(b * BN + c), r);
#pragma unroll
          for (int i = 0; i < 16; ++i) sum[c + i] += __uint_as_float(r[i]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.acc_empty[b]);
      }
      if (kt < blocks) break;
      const int m0 = tile_m0(t) + q * 32, n0 = tile_n0(t) + half * COLS;
      unsigned any_bad = 0;
#pragma unroll
      for (int c = 0; c < COLS; c += 16) {             // 64 bytes of each row at a time
#pragma unroll
        for (int p = 0; p < 4; ++p)
          stg[stage_index(lane, p)] = make_uint4(__float_as_uint(sum[c + 4 * p]), __float_as_uint(sum[c + 4 * p + 1]),
                                                 __float_as_uint(sum[c + 4 * p + 2]), __float_as_uint(sum[c + 4 * p + 3]));
        __syncwarp();
        const int n = n0 + c + o_piece * 4;
        float bs[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) bs[e] = bias != nullptr && n + e < N ? bias[n + e] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {                  // four lanes on a row's 64 bytes, eight rows an instruction
          const int m = m0 + 8 * j + o_row;
          const uint4 u = stg[stage_index(8 * j + o_row, o_piece)];
          float v[4] = {__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w)};
          const bool fine = fabsf(v[0]) < INFINITY && fabsf(v[1]) < INFINITY && fabsf(v[2]) < INFINITY && fabsf(v[3]) < INFINITY;
          const unsigned bad = __ballot_sync(0xffffffffu, !fine && m < M && n < N);
          if (lane == 0) sm.bad[warp - SPLIT_WARPS][c / 4 + j] = bad;
          any_bad |= bad;
          if (m >= M || n >= N || !fine) continue;
          const size_t o = (size_t)m * ldc + n;
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = activate<EPI, false>(v[e] + bs[e]);
          if (n + 4 <= N && (o & 3) == 0) {
            if (residual != nullptr) {
              const float4 rr = *reinterpret_cast<const float4*>(residual + o);
              v[0] += rr.x; v[1] += rr.y; v[2] += rr.z; v[3] += rr.w;
            }
            *reinterpret_cast<float4*>(C + o) = make_float4(v[0], v[1], v[2], v[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n + e < N) C[o + e] = residual != nullptr ? v[e] + residual[o + e] : v[e];
          }
        }
        __syncwarp();                                  // the pieces are read before the next ones overwrite them
      }
      // What is not finite, after all the others: the sums need no registers any more (a call in the loop above cost every call 5 %).
      for (int piece = 0; any_bad && piece < COLS / 4; ++piece)
        for (unsigned bad = sm.bad[warp - SPLIT_WARPS][piece]; bad; bad &= bad - 1) {
          const int src = __ffs(bad) - 1, m = m0 + 8 * (piece & 3) + (src >> 2), n = n0 + (piece >> 2) * 16 + (src & 3) * 4;
          const float4 s = plain_dots(A + (size_t)m * lda, W + (size_t)n * K, min(4, N - n), K);
          if (lane < 4 && n + lane < N) {
            const size_t o = (size_t)m * ldc + n + lane;
            const float x = lane == 0 ? s.x : lane == 1 ? s.y : lane == 2 ? s.z : s.w;
            const float v = activate<EPI, false>(x + (bias != nullptr ? bias[n + lane] : 0.f));
            C[o] = residual != nullptr ? v + residual[o] : v;
          }
        }
      __syncwarp();
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  const bool aborted = sm.abort_flag != 0;
  if (threadIdx.x == 0 && aborted) atomicOr(status, MLXB_ST_WAIT_TIMEOUT);
  if (warp == MMA_WARP) {
    if (aborted && elect_one()) {      // products in flight may still write the tensor memory that is freed below
      umma_commit(&sm.drained);
      const uint32_t addr = smem_u32(&sm.drained);
      for (uint32_t p = 0; p < (1u << 20); ++p) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(addr), "r"(0u) : "memory");
        if (done) break;
      }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------- host side

template <int BN>
static int launch(const float* A, const float* W, const float* bias, const float* residual, float* C, int M, int N, int K, int lda,
                  int ldc, int epi, int* status, cudaStream_t stream) {
  static_assert(sizeof(Smem<BN>) + 1024 <= 227 * 1024, "the parts of two blocks fit a CTA's shared memory");
  const size_t smem = sizeof(Smem<BN>) + 1024;
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int sms = mlxb_sm_count();
  const dim3 grid((unsigned)(tiles < sms ? tiles : sms));
  return dispatch_activation(epi, [&](auto e) {
    auto kernel = linear_split_kernel<BN, decltype(e)::value>;
    static SharedLimit limit;
    const cudaError_t err = limit.raise(kernel, smem);
    if (err != cudaSuccess) return mlxb_fail((int)err, "linear (float32 in parts): %zu bytes of shared memory: %s", smem, cudaGetErrorString(err));
    launch_pdl(kernel, grid, dim3(THREADS), smem, stream, A, W, bias, residual, C, M, N, K, lda, ldc, status);
    return mlxb_check_launch("linear (float32 in parts)");
  });
}

// All float32: A [M, K] at row stride lda, W [N, K] contiguous, bias [N] or null, residual [M, N] at row stride ldc or null (may
// alias C), C [M, N] at row stride ldc.  K and lda multiples of 4; A, W, C and the residual 16-byte aligned.  status: int32 word
// that receives MLXB_ST_WAIT_TIMEOUT if a bounded wait inside the kernel gives up.
MLXB_EXPORT int mlxb_linear_split(const float* A, const float* W, const float* bias, const float* residual, float* C, int M, int N,
                                  int K, int lda, int ldc, int epi, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (K & 3) || (lda & 3) || lda < K || ldc < N)
    return mlxb_fail(MLXB_BAD_ARG, "linear (float32 in parts): K %d and row stride %d must be multiples of 4 (ldc %d, N %d)", K, lda,
                     ldc, N);
  if (((uintptr_t)A | (uintptr_t)W | (uintptr_t)C | (uintptr_t)residual) & 15)
    return mlxb_fail(MLXB_BAD_ARG, "linear (float32 in parts): operands must be 16-byte aligned");
  const char* want = getenv("MLXB_SPLIT_BN");      // experiments and tests
  const long long rows = (M + BM - 1) / BM, sms = mlxb_sm_count();
  const long long wide = (rows * ((N + 127) / 128) + sms - 1) / sms, narrow = (rows * ((N + 63) / 64) + sms - 1) / sms;
  // Waves of wide tiles against waves of narrow ones, us: one and one 35 and 26 (64 x 3072 x 1024), two and three 65.7 and 64.3 (737 x
  // 4096 x 1024) and 92 and 94 (2048 x 1600 x 1600), two and four 65.8 and 84 (1024 x 4096 x 1024), three and six 93 and 120 (2048 x 3072
  // x 1024), one and two 33.5 and 42.3 (2048 x 1024 x 1024): the line lies where both take the same.
  const bool take_wide = want ? atoi(want) == 128 : wide * 100 <= narrow * 62;
  if (take_wide) return launch<128>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, status, stream);
  return launch<64>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, status, stream);
}
