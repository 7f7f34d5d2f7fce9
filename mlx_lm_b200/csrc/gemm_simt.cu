// Generic linear layer on the CUDA cores, true 32-bit arithmetic:
//   C[M,N] = epilogue(A[M,K] . W[N,K]^T + bias[N]) (+ residual[M,N])
// A and W are float32 or bfloat16 (one dtype for both); products and sums are
// float32 FMAs; C is that dtype or float32, and the residual has C's dtype.
// In the float32 engine these kernels take single rows, the output head and
// inner sizes below 128 (gemm_split.cu the rows of longer runs); they are the
// fallback of the bfloat16 engine for shapes its tensor-core kernels refuse.
//
// Every output element adds k in order within segments of SEG = 128, and the segments' sums in order: one order for
// every kernel, tile and number of rows, so a row's result does not depend on how many other rows the call has.  (A
// segment is what one warp of the few-rows kernel adds up alone; 128 dependent FMAs take 0.3 us, the 4096 of a long
// row 8 us.)
//
//   linear_tile   any M, N, K.  128 x 64 (or 64 x 64) outputs a block, 8 x 8 a thread: the loads of shared memory and the FMAs
//                 take about as long as one another (a warp's k: four 16-byte loads of four cycles, 32 instructions of
//                 two FMAs, fma.rn.f32x2, of 2.4), and two groups of warps, on segments in turns, fill an SM that gets a
//                 single tile.  1024 rows: 1024 x 1024 245 -> 70 us, 3072 x 1024 300 -> 208, 1024 x 4096 973 -> 264 (the
//                 64 x 64 tiles of 4 x 4 a thread that this replaces, which read global memory between two barriers):
//                 31 to 35 TFLOP/s of the 74 that the FMA pipes have.
//   linear_small  any M, N; one segment, or few outputs.  64 x 64 outputs a block of 256 threads, 4 x 4 a thread, the next K step on
//                 its way during this one's FMAs.  64 rows, 512 x 64: 6.0 us in float32, 6.2 in bfloat16.
//   linear_rows   float32, up to 16 rows, 16-byte rows: bound by the stream of W (one row: 206 MB in 70 us) and by latency.
//                 A warp takes 8 columns and a segment at a time; its W and A pieces travel by cp.async into memory of its
//                 own, the first of W before the wait for the kernel before.  One row: 1024 x 1024 70 -> 2.7 us,
//                 1024 x 4096 276 -> 6.8; 16 rows: 1024 x 4096 284 -> 15 us.
#include "activations.cuh"

MLXB_DEFINE_LAST_ERROR()

constexpr int SEG = 128;

// ---------------------------------------------------------------- tiles

constexpr int BN = 64, BK = 16;
static_assert(SEG % BK == 0, "a segment is a whole number of K steps");

typedef unsigned long long f32x2;      // two float32, the first in the low half

__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(f32x2& d, f32x2 a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ f32x2 twice(float v) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}

// Four neighbouring k of one row as they lie in memory, zeros outside the matrix; made float32 when they are stored, so that all
// loads of a thread are on their way together.  VEC: one access (K and the row stride multiples of 4, bases aligned to it).
template <typename T, bool VEC> struct Quad;
template <bool VEC>
struct Quad<float, VEC> {
  float4 v;
  __device__ __forceinline__ void load(const float* p, bool row_ok, int k, int K) {
    if (VEC) {
      v = row_ok && k < K ? *reinterpret_cast<const float4*>(p + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!row_ok) return;
      if (k < K) v.x = p[k];
      if (k + 1 < K) v.y = p[k + 1];
      if (k + 2 < K) v.z = p[k + 2];
      if (k + 3 < K) v.w = p[k + 3];
    }
  }
  __device__ __forceinline__ float4 value() const { return v; }
};
template <>
struct Quad<__nv_bfloat16, true> {
  uint2 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p, bool row_ok, int k, int K) {
    v = row_ok && k < K ? *reinterpret_cast<const uint2*>(p + k) : make_uint2(0u, 0u);
  }
  __device__ __forceinline__ float4 value() const {
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
  }
};
template <>
struct Quad<__nv_bfloat16, false> {
  unsigned v[4];
  __device__ __forceinline__ void load(const __nv_bfloat16* p, bool row_ok, int k, int K) {
    const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = row_ok && k + i < K ? u[k + i] : 0u;
  }
  __device__ __forceinline__ float4 value() const {
    return make_float4(__uint_as_float(v[0] << 16), __uint_as_float(v[1] << 16), __uint_as_float(v[2] << 16), __uint_as_float(v[3] << 16));
  }
};

// Two groups of BM threads take the segments in turns, each through tiles of its own; the second hands its sums to the
// first, which adds them up in order.
template <int BM>
struct TileMemory {
  static constexpr int LDA = BM + 4, LDW = BN + 4;
  float a[2][2][BK][LDA];                // [group][stage][k][row]
  float w[2][2][BK][LDW];                // [group][stage][k][column]
  f32x2 sums[2][32][BM];                 // [pair of segments & 1][value][thread of the second group]
};

template <typename T, typename TO, int EPI, int BM, bool VEC>
__global__ void __launch_bounds__(BM * 2, 128 / BM)
linear_tile_kernel(const T* A, const T* __restrict__ W, const float* __restrict__ bias, const TO* residual, TO* C, int M,
                   int N, int K, int lda, int ldc) {
  constexpr int AQ = 4, WQ = BN * 4 / BM;      // float4 pieces a thread fetches a step
  extern __shared__ __align__(16) char tile_sm[];
  TileMemory<BM>& sm = *reinterpret_cast<TileMemory<BM>*>(tile_sm);
  const int group = threadIdx.x / BM, tid = threadIdx.x % BM, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // Rows 4 ty .. + 3 and BM/2 + 4 ty .. + 3, columns 4 tx .. + 3 and 32 + 4 tx .. + 3: a 16-byte load of eight
  // neighbouring lanes covers 128 bytes of W or one address of A.
  const int tx = lane & 7, ty = (lane >> 3) + 4 * warp;
  // A warp fetches 16 rows by 8 k: whole sectors, and stores of 32 different banks.
  const int lr = (lane & 15) + 16 * (warp >> 1), lk = 4 * ((lane >> 4) + 2 * (warp & 1));
  Quad<T, VEC> aq[AQ], wq[WQ];
  auto fetch_w = [&](int k0) {
#pragma unroll
    for (int i = 0; i < WQ; ++i) {
      const int n = n0 + lr + i * (BM / 4);
      wq[i].load(W + (size_t)n * K, n < N, k0 + lk, K);
    }
  };
  auto fetch_a = [&](int k0) {
#pragma unroll
    for (int i = 0; i < AQ; ++i) {
      const int m = m0 + lr + i * (BM / 4);
      aq[i].load(A + (size_t)m * lda, m < M, k0 + lk, K);
    }
  };
  auto put = [&](int b) {
#pragma unroll
    for (int i = 0; i < AQ; ++i) {
      float (*d)[TileMemory<BM>::LDA] = sm.a[group][b];
      const int r = lr + i * (BM / 4);
      const float4 v = aq[i].value();
      d[lk][r] = v.x; d[lk + 1][r] = v.y; d[lk + 2][r] = v.z; d[lk + 3][r] = v.w;
    }
#pragma unroll
    for (int i = 0; i < WQ; ++i) {
      float (*d)[TileMemory<BM>::LDW] = sm.w[group][b];
      const int c = lr + i * (BM / 4);
      const float4 v = wq[i].value();
      d[lk][c] = v.x; d[lk + 1][c] = v.y; d[lk + 2][c] = v.z; d[lk + 3][c] = v.w;
    }
  };
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(BM) : "memory"); };
  f32x2 acc[4][8], tot[4][8];                  // [pair of rows][column]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = tot[i][j] = 0ull;
  fetch_w(group * SEG);
  pdl_wait();
  pdl_trigger();
  A = after_wait(A);
  residual = after_wait(residual);
  fetch_a(group * SEG);
  put(0);
  group_sync();
  int b = 0;
  const int pairs = (K + 2 * SEG - 1) / (2 * SEG);
  for (int p = 0; p < pairs; ++p) {
    const int begin = (2 * p + group) * SEG, end = min(begin + SEG, K);
    for (int k0 = begin; k0 < end; k0 += BK) {
      const int next = k0 + BK < end ? k0 + BK : begin + 2 * SEG;     // the group's next segment follows its last step
      const bool more = next < K;
      if (more) {
        fetch_w(next);
        fetch_a(next);
      }
      const float* pa = &sm.a[group][b][0][4 * ty];
      const float* pw = &sm.w[group][b][0][4 * tx];
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(pa + kk * TileMemory<BM>::LDA);
        const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(pa + kk * TileMemory<BM>::LDA + BM / 2);
        const float4 w0 = *reinterpret_cast<const float4*>(pw + kk * TileMemory<BM>::LDW);
        const float4 w1 = *reinterpret_cast<const float4*>(pw + kk * TileMemory<BM>::LDW + 32);
        const f32x2 a[4] = {a0.x, a0.y, a1.x, a1.y};
        const f32x2 w[8] = {twice(w0.x), twice(w0.y), twice(w0.z), twice(w0.w), twice(w1.x), twice(w1.y), twice(w1.z), twice(w1.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) fma2(acc[i][j], a[i], w[j]);
      }
      if (more) {
        b ^= 1;
        put(b);
        group_sync();
      }
    }
    if (group == 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) sm.sums[p & 1][i * 8 + j][tid] = acc[i][j];
    }
    __syncthreads();      // two buffers: the second group's next sums do not touch what the first still reads
    if (group == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          add2(tot[i][j], acc[i][j]);
          add2(tot[i][j], sm.sums[p & 1][i * 8 + j][tid]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  }
  if (group == 1) return;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int m = m0 + (i & 2 ? BM / 2 : 0) + 4 * ty + 2 * (i & 1) + e;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int n = n0 + (j & 4 ? 32 : 0) + 4 * tx + (j & 3);
        if (n >= N) continue;
        float v = __uint_as_float((unsigned)(e ? tot[i][j] >> 32 : tot[i][j]));
        if (bias) v += bias[n];
        v = activate<EPI, false>(v);
        if (residual) v += to_f(residual[(size_t)m * ldc + n]);
        C[(size_t)m * ldc + n] = from_f<TO>(v);
      }
    }
}

// ---------------------------------------------------------------- small products

// Bound by the chain of K steps.  64 x 64 outputs a block of 256 threads, 4 x 4 a thread, two K steps in shared memory: the tiles
// above have half of their threads without work when there is one segment, and four times as much for a thread to fetch a step.
template <typename T, typename TO, int EPI, bool VEC>
__global__ void __launch_bounds__(256)
linear_small_kernel(const T* A, const T* __restrict__ W, const float* __restrict__ bias, const TO* residual, TO* C, int M, int N,
                    int K, int lda, int ldc) {
  __shared__ __align__(16) float sa[2][BK][64 + 4];
  __shared__ __align__(16) float sw[2][BK][BN + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;      // rows 4 ty .., columns 4 tx ..
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * BN;
  const int lr = tid >> 2, lk = (tid & 3) * 4;                    // a thread fetches four k of one row of A and of W
  const bool m_in = m0 + lr < M, n_in = n0 + lr < N;
  const T* w_row = W + (size_t)(n_in ? n0 + lr : 0) * K;
  Quad<T, VEC> aq, wq;
  wq.load(w_row, n_in, lk, K);
  pdl_trigger();
  pdl_wait();
  A = after_wait(A);
  residual = after_wait(residual);
  const T* a_row = A + (size_t)(m_in ? m0 + lr : 0) * lda;
  auto put = [&](int b) {
    const float4 a = aq.value(), w = wq.value();
    sa[b][lk][lr] = a.x; sa[b][lk + 1][lr] = a.y; sa[b][lk + 2][lr] = a.z; sa[b][lk + 3][lr] = a.w;
    sw[b][lk][lr] = w.x; sw[b][lk + 1][lr] = w.y; sw[b][lk + 2][lr] = w.z; sw[b][lk + 3][lr] = w.w;
  };
  float tot[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) tot[i][j] = 0.f;
  aq.load(a_row, m_in, lk, K);
  put(0);
  __syncthreads();
  int b = 0;
  for (int s0 = 0; s0 < K; s0 += SEG) {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const int end = min(s0 + SEG, K);
    for (int k0 = s0; k0 < end; k0 += BK) {
      const bool more = k0 + BK < K;
      if (more) {
        wq.load(w_row, n_in, k0 + BK + lk, K);
        aq.load(a_row, m_in, k0 + BK + lk, K);
      }
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        const float4 a = *reinterpret_cast<const float4*>(&sa[b][kk][ty * 4]), w = *reinterpret_cast<const float4*>(&sw[b][kk][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
      }
      if (more) {
        b ^= 1;
        put(b);
        __syncthreads();
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) tot[i][j] += acc[i][j];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + 4 * ty + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + 4 * tx + j;
      if (n >= N) continue;
      float v = tot[i][j];
      if (bias) v += bias[n];
      v = activate<EPI, false>(v);
      if (residual) v += to_f(residual[(size_t)m * ldc + n]);
      C[(size_t)m * ldc + n] = from_f<TO>(v);
    }
  }
}

// ---------------------------------------------------------------- few rows

constexpr int RW_COLS = 8, RW_LD = SEG + 4;             // columns a block takes; floats between rows in shared memory
constexpr int rw_warps(int R) { return R > 2 ? 4 : 8; } // warps a block has at most: two pieces each have to fit the SM

__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

// R: rows a lane adds up (rows lane/8, lane/8 + 4, ...: up to 4 R rows in all).
template <int EPI, int R>
__global__ void __launch_bounds__(32 * rw_warps(R))
linear_rows_kernel(const float* A, const float* __restrict__ W, const float* __restrict__ bias, const float* residual,
                   float* C, int M, int N, int K, int lda, int ldc) {
  extern __shared__ __align__(16) float rw_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int n0 = blockIdx.x * RW_COLS, nseg = (K + SEG - 1) / SEG;
  constexpr int BUF = (RW_COLS + 4 * R) * RW_LD;            // one piece: 8 rows of W, 4 R rows of A
  float* part = rw_sm;                                      // [nseg][4 R][8]
  float* mine = rw_sm + nseg * 4 * R * RW_COLS + warp * 2 * BUF;
  auto ask_w = [&](int s, float* buf) {
    const int k = s * SEG + 4 * lane;
#pragma unroll
    for (int c = 0; c < RW_COLS; ++c) {
      const bool ok = n0 + c < N && k < K;
      cp16(buf + c * RW_LD + 4 * lane, W + (ok ? (size_t)(n0 + c) * K + k : 0), ok);
    }
  };
  auto ask_a = [&](int s, float* buf) {
    const int k = s * SEG + 4 * lane;
#pragma unroll
    for (int m = 0; m < 4 * R; ++m)
      if (m < M) cp16(buf + (RW_COLS + m) * RW_LD + 4 * lane, A + (k < K ? (size_t)m * lda + k : 0), k < K);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (warp < nseg) ask_w(warp, mine);
  pdl_wait();
  pdl_trigger();
  A = after_wait(A);
  residual = after_wait(residual);
  if (warp < nseg) ask_a(warp, mine);
  const int col = lane & 7, row = lane >> 3;
  int b = 0;
  for (int s = warp; s < nseg; s += nw) {
    float* buf = mine + b * BUF;
    b ^= 1;
    if (s + nw < nseg) {
      ask_w(s + nw, mine + b * BUF);
      ask_a(s + nw, mine + b * BUF);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    float acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.f;
    const float* pw = buf + col * RW_LD;
    const float* pa = buf + (RW_COLS + row) * RW_LD;
    // beyond K the copies left zeros in W and in A: they add nothing
#pragma unroll 8
    for (int k = 0; k < SEG; k += 4) {
      const float4 w = *reinterpret_cast<const float4*>(pw + k);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(pa + i * 4 * RW_LD + k);
        acc[i] = fmaf(a.x, w.x, acc[i]);
        acc[i] = fmaf(a.y, w.y, acc[i]);
        acc[i] = fmaf(a.z, w.z, acc[i]);
        acc[i] = fmaf(a.w, w.w, acc[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) part[(s * 4 * R + row + 4 * i) * RW_COLS + col] = acc[i];
    __syncwarp();
  }
  __syncthreads();
  for (int e = tid; e < M * RW_COLS; e += blockDim.x) {
    const int m = e / RW_COLS, n = n0 + e % RW_COLS;
    if (n >= N) continue;
    float v = 0.f;
    for (int s = 0; s < nseg; ++s) v += part[s * 4 * R * RW_COLS + e];
    if (bias) v += bias[n];
    v = activate<EPI, false>(v);
    if (residual) v += residual[(size_t)m * ldc + n];
    C[(size_t)m * ldc + n] = v;
  }
}

// ---------------------------------------------------------------- launch

// 16 rows: beyond, every block's copies of A outweigh those of W (17 rows of 1024 x 1024 take the tiles 44 us, 16 rows
// here 6); K: the segments' sums have to fit shared memory beside the pieces.
constexpr int RW_MAX_ROWS = 16, RW_MAX_K = 16384;

static constexpr size_t rows_memory(int R, int nseg, int warps) {
  return sizeof(float) * (size_t)(nseg * 4 * R * RW_COLS + warps * 2 * (RW_COLS + 4 * R) * RW_LD);
}

template <int R>
static int launch_rows(const float* A, const float* W, const float* bias, const float* residual, float* C, int M, int N, int K,
                       int lda, int ldc, int epi, cudaStream_t stream) {
  const int nseg = (K + SEG - 1) / SEG, warps = nseg < rw_warps(R) ? nseg : rw_warps(R);
  const size_t smem = rows_memory(R, nseg, warps);
  return dispatch_activation(epi, [&](auto e) {
    auto kernel = linear_rows_kernel<decltype(e)::value, R>;
    if (smem > 48 * 1024) {
      static SharedLimit limit;
      constexpr int WARPS = rw_warps(R), SEGS = RW_MAX_K / SEG;
      const cudaError_t err = limit.raise(kernel, rows_memory(R, SEGS, WARPS));
      if (err != cudaSuccess) return mlxb_fail((int)err, "linear: %zu bytes of shared memory: %s", smem, cudaGetErrorString(err));
    }
    launch_pdl(kernel, dim3((N + RW_COLS - 1) / RW_COLS), dim3(32 * warps), smem, stream, A, W, bias, residual, C, M, N, K, lda, ldc);
    return mlxb_check_launch("linear (few rows, float32)");
  });
}

template <typename T, typename TO, int BM, bool VEC>
static int launch_tile(const void* A, const void* W, const float* bias, const void* residual, void* C, int M, int N,
                       int K, int lda, int ldc, int epi, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  return dispatch_activation(epi, [&](auto e) {
    auto kernel = linear_tile_kernel<T, TO, decltype(e)::value, BM, VEC>;
    static SharedLimit limit;
    const cudaError_t err = limit.raise(kernel, sizeof(TileMemory<BM>));
    if (err != cudaSuccess) return mlxb_fail((int)err, "linear: %zu bytes of shared memory: %s", sizeof(TileMemory<BM>), cudaGetErrorString(err));
    launch_pdl(kernel, grid, dim3(BM * 2), sizeof(TileMemory<BM>), stream, (const T*)A, (const T*)W, bias, (const TO*)residual,
               (TO*)C, M, N, K, lda, ldc);
    return mlxb_check_launch("linear (generic)");
  });
}

template <typename T, typename TO, bool VEC>
static int launch_small(const void* A, const void* W, const float* bias, const void* residual, void* C, int M, int N, int K,
                        int lda, int ldc, int epi, cudaStream_t stream) {
  const dim3 grid((N + BN - 1) / BN, (M + 63) / 64);
  return dispatch_activation(epi, [&](auto e) {
    launch_pdl(linear_small_kernel<T, TO, decltype(e)::value, VEC>, grid, dim3(256), 0, stream, (const T*)A, (const T*)W, bias,
               (const TO*)residual, (TO*)C, M, N, K, lda, ldc);
    return mlxb_check_launch("linear (generic, small)");
  });
}

template <typename T, typename TO, bool VEC>
static int launch(const void* A, const void* W, const float* bias, const void* residual, void* C, int M, int N,
                  int K, int lda, int ldc, int epi, cudaStream_t stream) {
  // Small products first: one segment, or few tiles of up to 320 (64 rows, bfloat16 and float32: 512 x 64 6.2 and 6.0 us here, 10.4
  // and 9.8 on the tiles; 96 x 320 20.2 and 18.1, on the tiles 22.2 and 20.2; 1024 x 1024 59 and 52, on the tiles 54 and 48).
  // On the tiles an SM works at a rate that hardly depends on their size, so what counts is the most rows of 64 x 64
  // outputs that one SM gets; at a tie the larger tile reads less.
  const long long cols = (N + BN - 1) / BN, sms = mlxb_sm_count(), tiles = (M + 63) / 64 * cols;
  if (K <= SEG || (K <= 320 && tiles <= sms))
    return launch_small<T, TO, VEC>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
  const long long large = 2 * (((M + 127) / 128 * cols + sms - 1) / sms), small = (tiles + sms - 1) / sms;
  if (large <= small) return launch_tile<T, TO, 128, VEC>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
  return launch_tile<T, TO, 64, VEC>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
}

// dtype: dtype of A and W.  out_f32 != 0: C and the residual are float32 whatever dtype is.
// lda: row stride of A in elements (>= K); ldc: row stride of C and residual.
// bias (float32[N]) and residual may be null.
MLXB_EXPORT int mlxb_linear_simt(int dtype, int out_f32, const void* A, const void* W, const float* bias,
                                 const void* residual, void* C, int M, int N, int K, int lda, int ldc, int epi,
                                 cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldc < N) return mlxb_fail(MLXB_BAD_ARG, "linear: K %d lda %d ldc %d N %d", K, lda, ldc, N);
  if ((M + 63) / 64 > 65535) return mlxb_fail(MLXB_BAD_ARG, "linear: %d rows are too many for one call", M);
  if (dtype == MLXB_F32) {
    const bool vec = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    if (vec && M <= RW_MAX_ROWS && K <= RW_MAX_K) {
      const float *a = (const float*)A, *w = (const float*)W, *r = (const float*)residual;
      if (M <= 4) return launch_rows<1>(a, w, bias, r, (float*)C, M, N, K, lda, ldc, epi, stream);
      if (M <= 8) return launch_rows<2>(a, w, bias, r, (float*)C, M, N, K, lda, ldc, epi, stream);
      return launch_rows<4>(a, w, bias, r, (float*)C, M, N, K, lda, ldc, epi, stream);
    }
    if (vec) return launch<float, float, true>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
    return launch<float, float, false>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
  }
  if (dtype == MLXB_BF16) {
    const bool vec = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 7) == 0;
    if (vec && out_f32) return launch<__nv_bfloat16, float, true>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
    if (vec) return launch<__nv_bfloat16, __nv_bfloat16, true>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
    if (out_f32) return launch<__nv_bfloat16, float, false>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
    return launch<__nv_bfloat16, __nv_bfloat16, false>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, stream);
  }
  return mlxb_fail(MLXB_BAD_DTYPE, "linear: dtype code %d", dtype);
}
