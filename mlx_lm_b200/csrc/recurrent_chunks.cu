// Runs of rows through the recurrences with a state of fixed size (recurrent.cu), 64 rows at a time on tensor cores.
//
// Token by token a scan is a chain as long as the run: 1024 rows of the state-space layer (32 heads of 64 columns, 128 rows of
// state, two requests) took 387 us and of the gated delta rule (16 heads of 64 x 64) 423, with almost everything idle; in
// chunks they take 107 and 159, the delta rule in two passes 106 (eight runs of 100 rows: 107 -> 59 and 54 -> 43; one of 70: 24 -> 15 and 33 -> 21).  A chunk
// takes its time however few rows it has, and a block most of an SM's shared memory, so short runs, and many states of the
// delta rule, stay with the scan (ops.chunk_rule).  A block of threads here has a (request, head, slice of VS columns of the
// state), keeps its state in registers as accumulators and walks the run in chunks of 64 rows; within a chunk everything is
// a product of small matrices.  What is left is a chain too, of a chunk's phases.
//
// Nothing is held in less than 32 bits.  Inputs are bfloat16 as they come; every float32 operand of a product (the state,
// decay-weighted scores, weighted inputs) goes in as three bfloat16 numbers whose sum it is, the smallest first.  Decays
// are differences of a sum of logarithms that is kept in 64 bits, so that neighbours late in a chunk lose nothing.  Against
// 64 bits, with decays as the layers' random weights have them, outputs are 1.0e-7 (the scan 1.05e-7) and 1.3e-7 off (1.3e-7), states
// after a run 0.8e-7 (0.7e-7) and 1.1e-7 (0.9e-7); with slow decays, e.g. dt_bias 6 less and 1024 rows, outputs 0.5e-7 (6.2e-7)
// and 1.8e-7 (8.6e-7), states 1.1e-7 (23e-7) and 1.6e-7 (9.0e-7).
#include "common.cuh"
#include "mma_bf16.cuh"
#include "recurrent_tiles.cuh"

MLXB_DEFINE_LAST_ERROR()

__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

constexpr int RC_Q = 64;            // rows of a chunk
constexpr int RC_THREADS = 256;

// x as the sum of three bfloat16 numbers.  What is not finite (and what is above bfloat16's largest number, 0.996 of float32's)
// is the first of them, beside zeros: a product with it is then what a product with x would be.
__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
  a = __float2bfloat16_rn(x);
  float r = x - __bfloat162float(a);
  r = fabsf(r) < INFINITY ? r : 0.f;
  b = __float2bfloat16_rn(r);
  c = __float2bfloat16_rn(r - __bfloat162float(b));
}
// two neighbours of a row into the three planes (plane: elements between them)
__device__ __forceinline__ void store_split(__nv_bfloat16* dst, int plane, float x, float y) {
  __nv_bfloat162 p[3];
  split3(x, p[0].x, p[1].x, p[2].x);
  split3(y, p[0].y, p[1].y, p[2].y);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<__nv_bfloat162*>(dst + i * plane) = p[i];
}

// d += A B with the sum rounded to nearest: the tensor core cuts off what it adds to its accumulator, which over a chain of
// products leaves twice the error of a scan in float32.  The planes of lower order may stay in the tensor core's accumulator.
__device__ __forceinline__ void mma_add(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
  mb_mma(t, a, b0, b1);
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] += t[i];
}
__device__ __forceinline__ void mma_plane(float (&d)[4], float (&low)[4], int plane, const unsigned (&a)[4], unsigned b0, unsigned b1) {
  if (plane == 0) mma_add(d, a, b0, b1);
  else mb_mma(low, a, b0, b1);
}

// Fragments from shared memory at row stride ld (elements): A of rows x k, A stored as k x rows, B (16 columns, two tiles of 8)
// stored as columns x k, B stored as k x columns.
__device__ __forceinline__ void frag_a(unsigned (&r)[4], const __nv_bfloat16* p, int ld, int lane) {
  mb_ldmatrix(r, mb_smem(p + (lane & 15) * ld + (lane >> 4) * 8));
}
__device__ __forceinline__ void frag_a_t(unsigned (&r)[4], const __nv_bfloat16* p, int ld, int lane) {
  mb_ldmatrix_trans(r, mb_smem(p + ((lane & 7) + ((lane >> 4) & 1) * 8) * ld + ((lane >> 3) & 1) * 8));
}
__device__ __forceinline__ void frag_b(unsigned (&r)[4], const __nv_bfloat16* p, int ld, int lane) {
  mb_ldmatrix(r, mb_smem(p + ((lane & 7) + ((lane >> 4) & 1) * 8) * ld + ((lane >> 3) & 1) * 8));
}
__device__ __forceinline__ void frag_b_t(unsigned (&r)[4], const __nv_bfloat16* p, int ld, int lane) {
  mb_ldmatrix_trans(r, mb_smem(p + (lane & 15) * ld + (lane >> 4) * 8));
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool have) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(mb_smem(dst)), "l"(src), "r"(have ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// 64 rows of `width` columns (zeros beyond n rows and beyond `cols`) into [64][ld].  vec: 16-byte pieces are aligned and lie
// inside or outside as a whole (base, row stride and cols multiples of 8); their copies are asynchronous.
__device__ __forceinline__ void stage_rows(const __nv_bfloat16* src, int lds_src, int n, int cols, int width, __nv_bfloat16* dst, int ld,
                                           bool vec) {
  if (vec) {
    const int per = width / 8;
    for (int e = threadIdx.x; e < RC_Q * per; e += RC_THREADS) {
      const int row = e / per, c = (e - row * per) * 8;
      const bool have = row < n && c < cols;
      cp_async16(dst + row * ld + c, have ? src + (size_t)row * lds_src + c : src, have);
    }
  } else {
    for (int e = threadIdx.x; e < RC_Q * width; e += RC_THREADS) {
      const int row = e / width, c = e - row * width;
      dst[row * ld + c] = (row < n && c < cols) ? src[(size_t)row * lds_src + c] : __float2bfloat16_rn(0.f);
    }
  }
}

// The logarithm of a row's decay, from minus the rate and the step.  Below -200 a decay is zero in float32 whatever follows, so
// that an infinite step leaves sums with differences.
__device__ __forceinline__ double log_decay(float rate, float step) {
  const float l = rate * step;
  return (double)(l < -200.f ? -200.f : l);
}

// Inclusive sums over the chunk of one value a row, by one warp: lane l has rows 2 l and 2 l + 1.  A row's sum has only values
// of rows up to it (and no differences of later sums), so that a NaN stays behind the rows before it.
__device__ __forceinline__ void chunk_sums(double& a, double& b, int lane) {
  double t = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double u = __shfl_up_sync(0xffffffffu, t, o);
    if (lane >= o) t += u;
  }
  const double before = __shfl_up_sync(0xffffffffu, t, 1);
  if (lane > 0) a += before;
  b += a;
}

// Rows of a chunk that are not finite.  A row's weights for the rows behind it are zeros, and zero times an infinity is not
// zero: in a diagonal tile of 16 rows by 16 such values leave the product (drop_bad, from a B fragment of two neighbouring
// values each) and are added to the rows that have them behind them (add_bad).  The other values' sums stay as they are.
__device__ __forceinline__ void drop_bad(unsigned& u) {
  if ((u & 0x7f80u) == 0x7f80u) u &= 0xffff0000u;
  if ((u & 0x7f800000u) == 0x7f800000u) u &= 0x0000ffffu;
}
// value(s, c): row s, column c; p: the weights' planes, `plane` elements apart.  This thread's eight results of rows 16 ti ..,
// columns c16 .., as accumulators of two tiles.
template <typename Value>
__device__ __forceinline__ void add_bad(float (&acc)[2][4], const __nv_bfloat16* p, int plane, int ldp, int ti, int c16, int g, int q,
                                        Value value) {
#pragma unroll 1
  for (int s = 16 * ti; s < 16 * ti + 16; ++s)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 16 * ti + g + (e >> 1) * 8;
        const float v = value(s, c16 + 8 * j + 2 * q + (e & 1));
        if (s > t || fabsf(v) < INFINITY) continue;
        const __nv_bfloat16* w = p + t * ldp + s;
        acc[j][e] = fmaf(to_f(w[0]) + (to_f(w[plane]) + to_f(w[2 * plane])), v, acc[j][e]);
      }
}

// ---------------------------------------------------------------- state-space scan (Mamba-2)
// With L_t the sum of the logarithms of the decays up to row t, S_0 the state before the chunk:
//   y_t = exp(L_t) C_t . S_0 + sum_{s <= t} exp(L_t - L_s) dt_s (C_t . B_s) x_s + D x_t
//   S   = exp(L_end) S_0 + sum_s exp(L_end - L_s) dt_s B_s x_s^T
constexpr int M2_VS = 32;

template <int NP>
struct Mamba2Memory {
  static constexpr int LN = NP + 8, LV = M2_VS + 8, LP = RC_Q + 8;
  __nv_bfloat16 b[2][RC_Q * LN], c[2][RC_Q * LN], x[2][RC_Q * LV];      // two chunks: the next one is on its way
  __nv_bfloat16 state[3][M2_VS * LN];                                   // [column][row of the state]
  __nv_bfloat16 wx[3][RC_Q * LV];                                       // x_s times what is left of it at the chunk's end
  __nv_bfloat16 p[3][RC_Q * LP];                                        // [t][s]
  double sum[RC_Q];
  float dt[RC_Q], left[RC_Q], since[RC_Q];                              // step size, weight at the end, decay since the start
};

template <int NP>
__global__ void __launch_bounds__(RC_THREADS, NP > 64 ? 1 : 2)      // as many as their shared memory lets an SM hold
mamba2_chunks_kernel(const __nv_bfloat16* xbc, int ldx, int x_off, int b_off, int c_off, const __nv_bfloat16* dt_raw, int lddt,
                     const float* __restrict__ dt_bias, const float* __restrict__ A_log, const float* __restrict__ Dskip,
                     float* state, const int* __restrict__ slots, const int* __restrict__ token_req,
                     const int* __restrict__ req_first_token, const int* __restrict__ requests, ChunkRule rule, float* __restrict__ y,
                     int ldy, int H, int G, int N, int V, int vec) {
  extern __shared__ __align__(16) char rc_sm[];
  using Mem = Mamba2Memory<NP>;
  Mem& sm = *reinterpret_cast<Mem*>(rc_sm);
  constexpr int LN = Mem::LN, LV = Mem::LV, LP = Mem::LP;
  const int h = blockIdx.x, r = requests != nullptr ? requests[blockIdx.y] : (int)blockIdx.y, v0 = blockIdx.z * M2_VS;
  const int t0 = r >= 0 ? req_first_token[r] : 0, t1 = r >= 0 ? req_first_token[r + 1] : 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int grp = h / (H / G);
  pdl_trigger();
  const int n = run_length(token_req, t0, t1, r);
  if (!rule.chunks(n)) {                  // goes through the scan, or only fills the list of requests up
    pdl_wait();                           // dependents were let go above: a grid without runs must not end before its predecessor
    return;
  }
  // This warp's part of the state, as accumulators: columns v0 + 16 vi .., rows NP / 4 * ni .. of the state, in tiles of 8.
  constexpr int NT = NP / 32;
  const int vi = warp & 1, ni = warp >> 1;
  float S[NT][4];
  float* pool = state + ((size_t)slots[r] * H + h) * N * V;
  // older than this step: read before the wait (see recurrent.cu)
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int v = v0 + 16 * vi + g + (e >> 1) * 8, nn = (NP / 4) * ni + 8 * j + 2 * q + (e & 1);
      S[j][e] = (v < V && nn < N) ? pool[(size_t)v * N + nn] : 0.f;
    }
  const float negA = -expf(A_log[h]), skip = Dskip[h], bias = dt_bias[h];
  pdl_wait();
  xbc = after_wait(xbc);
  dt_raw = after_wait(dt_raw);
  auto fetch = [&](int buf, int c0) {
    const int nc = min(RC_Q, n - c0);
    const __nv_bfloat16* rows = xbc + (size_t)(t0 + c0) * ldx;
    stage_rows(rows + b_off + grp * N, ldx, nc, N, NP, sm.b[buf], LN, vec);
    stage_rows(rows + c_off + grp * N, ldx, nc, N, NP, sm.c[buf], LN, vec);
    stage_rows(rows + x_off + h * V + v0, ldx, nc, V - v0, M2_VS, sm.x[buf], LV, vec);
    cp_async_commit();
  };
  fetch(0, 0);
  for (int c0 = 0, buf = 0; c0 < n; c0 += RC_Q, buf ^= 1) {
    const int nc = min(RC_Q, n - c0);
    const __nv_bfloat16 *sb = sm.b[buf], *sc = sm.c[buf], *sx = sm.x[buf];
    cp_async_wait();
    // the chunk before has been read (its planes are written again below), this one's rows are there
    __syncthreads();
    if (warp == 0) {
      float d[2];
      double l[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = 2 * lane + i;
        d[i] = t < nc ? softplus_f(to_f(dt_raw[(size_t)(t0 + c0 + t) * lddt + h]) + bias) : 0.f;
        l[i] = log_decay(negA, d[i]);
      }
      chunk_sums(l[0], l[1], lane);
      const double end = __shfl_sync(0xffffffffu, l[1], 31);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = 2 * lane + i;
        sm.sum[t] = l[i];
        sm.dt[t] = d[i];
        sm.since[t] = expf((float)l[i]);
        sm.left[t] = expf((float)(end - l[i])) * d[i];
      }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        store_split(sm.state[0] + (16 * vi + g + (e >> 1) * 8) * LN + (NP / 4) * ni + 8 * j + 2 * q, M2_VS * LN, S[j][e], S[j][e + 1]);
    __syncthreads();
    if (c0 + RC_Q < n) fetch(buf ^ 1, c0 + RC_Q);
    bool bad = false;                        // a value of x that is not finite
    for (int e = tid; e < RC_Q * M2_VS / 2; e += RC_THREADS) {
      const int s = e / (M2_VS / 2), c = 2 * (e - s * (M2_VS / 2));
      const float2 xv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sx + s * LV + c));
      store_split(sm.wx[0] + s * LV + c, RC_Q * LV, sm.left[s] * xv.x, sm.left[s] * xv.y);
      bad |= !(fabsf(xv.x) < INFINITY && fabsf(xv.y) < INFINITY);
    }
    const int ti = warp >> 1;                // rows 16 ti .. of the chunk, for P and y
    // P: columns 32 (warp & 1) .., up to the diagonal's tile
#pragma unroll
    for (int pair = 0; pair < 2; ++pair) {
      const int s0 = 32 * (warp & 1) + 16 * pair;
      if (s0 > 16 * ti) continue;
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int k = 0; k < NP; k += 16) {
        unsigned a[4], bb[4];
        frag_a(a, sc + 16 * ti * LN + k, LN, lane);
        frag_b(bb, sb + s0 * LN + k, LN, lane);
        mma_add(acc[0], a, bb[0], bb[1]);
        mma_add(acc[1], a, bb[2], bb[3]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const int t = 16 * ti + g + (e >> 1) * 8, s = s0 + 8 * j + 2 * q;
          float w[2];
#pragma unroll
          for (int i = 0; i < 2; ++i)
            w[i] = s + i <= t ? expf((float)(sm.sum[t] - sm.sum[s + i])) * sm.dt[s + i] * acc[j][e + i] : 0.f;
          store_split(sm.p[0] + t * LP + s, RC_Q * LP, w[0], w[1]);
        }
    }
    bad = __syncthreads_or(bad);
    {   // y: columns 16 (warp & 1) .. of the slice
      const int c16 = 16 * (warp & 1);
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, low[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int pl = 2; pl >= 0; --pl)
#pragma unroll
        for (int k = 0; k < NP; k += 16) {
          unsigned a[4], bb[4];
          frag_a(a, sc + 16 * ti * LN + k, LN, lane);
          frag_b(bb, sm.state[pl] + c16 * LN + k, LN, lane);
          mma_plane(acc[0], low[0], pl, a, bb[0], bb[1]);
          mma_plane(acc[1], low[1], pl, a, bb[2], bb[3]);
        }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[j][e] = (acc[j][e] + low[j][e]) * sm.since[16 * ti + g + (e >> 1) * 8];
          low[j][e] = 0.f;
        }
      for (int k = 0; k <= 16 * ti; k += 16) {
        unsigned bb[4];
        frag_b_t(bb, sx + k * LV + c16, LV, lane);
        if (bad && k == 16 * ti) {
#pragma unroll
          for (int i = 0; i < 4; ++i) drop_bad(bb[i]);
        }
#pragma unroll
        for (int pl = 2; pl >= 0; --pl) {
          unsigned a[4];
          frag_a(a, sm.p[pl] + 16 * ti * LP + k, LP, lane);
          mma_plane(acc[0], low[0], pl, a, bb[0], bb[1]);
          mma_plane(acc[1], low[1], pl, a, bb[2], bb[3]);
        }
      }
      if (bad) add_bad(acc, sm.p[0], RC_Q * LP, LP, ti, c16, g, q, [&](int s, int c) { return to_f(sx[s * LV + c]); });
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = 16 * ti + g + (e >> 1) * 8, c = c16 + 8 * j + 2 * q + (e & 1);
          if (t < nc && v0 + c < V)
            y[(size_t)(t0 + c0 + t) * ldy + h * V + v0 + c] = fmaf(skip, to_f(sx[t * LV + c]), acc[j][e] + low[j][e]);
        }
    }
    const float keep = sm.since[RC_Q - 1];       // rows beyond the run decay nothing
    float add[NT][4], low[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) add[j][e] = low[j][e] = 0.f;
#pragma unroll
    for (int k = 0; k < RC_Q; k += 16) {
      unsigned a[3][4];
#pragma unroll
      for (int pl = 0; pl < 3; ++pl) frag_a_t(a[pl], sm.wx[pl] + k * LV + 16 * vi, LV, lane);
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        unsigned bb[4];
        frag_b_t(bb, sb + k * LN + (NP / 4) * ni + 8 * j, LN, lane);
#pragma unroll
        for (int pl = 2; pl >= 0; --pl) {
          mma_plane(add[j], low[j], pl, a[pl], bb[0], bb[1]);
          mma_plane(add[j + 1], low[j + 1], pl, a[pl], bb[2], bb[3]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf(keep, S[j][e], add[j][e] + low[j][e]);
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int v = v0 + 16 * vi + g + (e >> 1) * 8, nn = (NP / 4) * ni + 8 * j + 2 * q + (e & 1);
      if (v < V && nn < N) pool[(size_t)v * N + nn] = S[j][e];
    }
}

// The arguments of mlxb_mamba2_scan (bfloat16 inputs, states of up to 128 rows).  requests: the n_requests to look at (-1: none),
// or null for the first n_requests of the step; of these, the runs that the rule sends here.
MLXB_EXPORT int mlxb_mamba2_chunks(const void* xbc, int ldx, int x_off, int b_off, int c_off, const void* dt_raw, int lddt,
                                   const float* dt_bias, const float* A_log, const float* Dskip, float* state, const int* slots,
                                   const int* token_req, const int* req_first_token, float* y, int ldy, int H, int G, int N, int V,
                                   const int* requests, int n_requests, int scan_fixed, int scan_row, int chunk_fixed, int chunk_each,
                                   cudaStream_t stream) {
  if (n_requests <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || N <= 0 || V <= 0 || N > 128 || n_requests > 65535)
    return mlxb_fail(MLXB_BAD_ARG, "mamba2_chunks: %d heads in %d groups, state %d x %d (at most 128 rows)", H, G, N, V);
  const int vec = (((uintptr_t)xbc & 15) == 0 && ldx % 8 == 0 && x_off % 8 == 0 && b_off % 8 == 0 && c_off % 8 == 0 && N % 8 == 0 &&
                   V % 8 == 0);
  const dim3 grid(H, n_requests, (V + M2_VS - 1) / M2_VS);
  static SharedLimit limits[2];
  auto go = [&](auto kern, size_t smem, SharedLimit& limit) {
    const cudaError_t e = limit.raise(kern, smem);
    if (e != cudaSuccess) return mlxb_fail((int)e, "mamba2_chunks: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    launch_pdl(kern, grid, dim3(RC_THREADS), smem, stream, (const __nv_bfloat16*)xbc, ldx, x_off, b_off, c_off,
               (const __nv_bfloat16*)dt_raw, lddt, dt_bias, A_log, Dskip, state, slots, token_req, req_first_token, requests,
               ChunkRule{scan_fixed, scan_row, chunk_fixed, chunk_each}, y, ldy, H, G, N, V, vec);
    return mlxb_check_launch("mamba2_chunks");
  };
  if (N <= 64) return go(mamba2_chunks_kernel<64>, sizeof(Mamba2Memory<64>), limits[0]);
  return go(mamba2_chunks_kernel<128>, sizeof(Mamba2Memory<128>), limits[1]);
}

// ---------------------------------------------------------------- gated delta rule
// With G_t the product of the decays up to row t, S_0 the state before the chunk, k and q the unit vectors, the rows u of
// all updates of a chunk solve a triangular system:
//   (I + M) U = R,  M[t, s] = beta_t G_t / G_s (k_t . k_s) for s < t,  R_t = beta_t (v_t - G_t k_t . S_0)
//   o_t = G_t q_t . S_0 + sum_{s <= t} G_t / G_s (q_t . k_s) u_s,     S = G_end S_0 + sum_s G_end / G_s k_s u_s^T
// It is solved by blocks of 16 rows in float32: the four diagonal blocks are inverted side by side, then every block's
// rows follow from a product with its inverse and are taken out of the rows below.
constexpr int GD_VS = 32, GD_KP = 64;

struct DeltaMemory {
  static constexpr int LK = GD_KP + 8, LV = GD_VS + 8, LP = RC_Q + 8, LM = RC_Q + 4, LI = 20;
  __nv_bfloat16 k[2][RC_Q * LK], q[2][RC_Q * LK], v[2][RC_Q * LV];
  __nv_bfloat16 state[3][GD_VS * LK];            // [column][row of the state]
  __nv_bfloat16 p[3][RC_Q * LP];                 // [t][s]
  __nv_bfloat16 u[3][RC_Q * LV], wu[3][RC_Q * LV];      // the updates, and times what is left of them at the chunk's end
  float m[RC_Q * LM];                            // [t][s]
  float inv[4][16 * LI];
  float r[RC_Q * GD_VS];                         // right sides, then the updates
  double sum[RC_Q];
  float since[RC_Q], left[RC_Q], beta[RC_Q], rk[RC_Q], rq[RC_Q];
};

// What a chunk's rows have by themselves: decays and their sums (warp 0), what makes k and q unit vectors (warps 1 to 4).  a_raw, b_raw:
// this head's number in the chunk's first row.
template <typename Memory>
__device__ __forceinline__ void delta_rows(Memory& sm, const __nv_bfloat16* sk, const __nv_bfloat16* sq, const __nv_bfloat16* a_raw, int lda,
                                           const __nv_bfloat16* b_raw, int ldb, int nc, float negA, float bias, float q_scale) {
  constexpr int LK = Memory::LK;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (warp == 0) {
    double l[2];
    float beta[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      const size_t row = t;
      l[i] = t < nc ? log_decay(negA, softplus_f(to_f(a_raw[row * lda]) + bias)) : 0.;
      beta[i] = t < nc ? 1.f / (1.f + expf(-to_f(b_raw[row * ldb]))) : 0.f;
    }
    chunk_sums(l[0], l[1], lane);
    const double end = __shfl_sync(0xffffffffu, l[1], 31);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      sm.sum[t] = l[i];
      sm.beta[t] = beta[i];
      sm.since[t] = expf((float)l[i]);
      sm.left[t] = expf((float)(end - l[i]));
    }
  } else if (warp <= 4) {      // what makes k and q unit vectors, a thread a row
    const int t = (tid - 32) & 63;
    const bool keys = tid < 32 + 64;
    const uint4* row = reinterpret_cast<const uint4*>((keys ? sk : sq) + t * LK);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < GD_KP / 8; ++i) {
      float f[8];
      unpack8(row[i], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) sum = fmaf(f[e], f[e], sum);
    }
    if (keys) sm.rk[t] = 1.f / sqrtf(sum + 1e-6f);
    else sm.rq[t] = q_scale / sqrtf(sum + 1e-6f);
  }
}

// M into sm.m and P's three numbers into the planes at p.  ak, aq: this warp's 16 rows of k and of q.
template <typename Memory>
__device__ __forceinline__ void delta_scores(Memory& sm, const __nv_bfloat16* sk, const unsigned (&ak)[GD_KP / 16][4],
                                             const unsigned (&aq)[GD_KP / 16][4], __nv_bfloat16* p, int ldp, int plane) {
  constexpr int LK = Memory::LK, LM = Memory::LM;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3, ti = warp >> 1;
  // M and P: columns 32 (warp & 1) .., up to the diagonal's tile
#pragma unroll
  for (int pair = 0; pair < 2; ++pair) {
    const int s0 = 32 * (warp & 1) + 16 * pair;
    if (s0 > 16 * ti) continue;
    float kk[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, qk[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int k = 0; k < GD_KP / 16; ++k) {
      unsigned bb[4];
      frag_b(bb, sk + s0 * LK + 16 * k, LK, lane);
      mma_add(kk[0], ak[k], bb[0], bb[1]);
      mma_add(kk[1], ak[k], bb[2], bb[3]);
      mma_add(qk[0], aq[k], bb[0], bb[1]);
      mma_add(qk[1], aq[k], bb[2], bb[3]);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int t = 16 * ti + g + (e >> 1) * 8, s = s0 + 8 * j + 2 * q;
        float w[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float d = s + i <= t ? expf((float)(sm.sum[t] - sm.sum[s + i])) * sm.rk[s + i] : 0.f;
          w[i] = s + i <= t ? d * sm.rq[t] * qk[j][e + i] : 0.f;
          sm.m[t * LM + s + i] = s + i < t ? d * sm.beta[t] * sm.rk[t] * kk[j][e + i] : 0.f;
        }
        store_split(p + t * ldp + s, plane, w[0], w[1]);
      }
  }
}

__global__ void __launch_bounds__(RC_THREADS)
gated_delta_chunks_kernel(const __nv_bfloat16* qkv, int ldq, int q_off, int k_off, int v_off, const __nv_bfloat16* b_raw, int ldb,
                          const __nv_bfloat16* a_raw, int lda, const float* __restrict__ dt_bias, const float* __restrict__ A_log,
                          float* state, const int* __restrict__ slots, const int* __restrict__ token_req,
                          const int* __restrict__ req_first_token, const int* __restrict__ requests, ChunkRule rule,
                          float* __restrict__ o, int ldo, int H, int G, int K, int V, int vec) {
  extern __shared__ __align__(16) char rc_sm[];
  DeltaMemory& sm = *reinterpret_cast<DeltaMemory*>(rc_sm);
  constexpr int LK = DeltaMemory::LK, LV = DeltaMemory::LV, LP = DeltaMemory::LP, LM = DeltaMemory::LM, LI = DeltaMemory::LI;
  const int h = blockIdx.x, r = requests != nullptr ? requests[blockIdx.y] : (int)blockIdx.y, v0 = blockIdx.z * GD_VS;
  const int t0 = r >= 0 ? req_first_token[r] : 0, t1 = r >= 0 ? req_first_token[r + 1] : 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int grp = h / (H / G);
  pdl_trigger();
  const int n = run_length(token_req, t0, t1, r);
  if (!rule.chunks(n)) {
    pdl_wait();
    return;
  }
  // this warp's part of the state, as accumulators: columns v0 + 16 vi .., rows 16 ni .. of the state, in tiles of 8
  const int vi = warp & 1, ni = warp >> 1;
  float S[2][4];
  float* pool = state + ((size_t)slots[r] * H + h) * K * V;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int v = v0 + 16 * vi + g + (e >> 1) * 8, kk = 16 * ni + 8 * j + 2 * q + (e & 1);
      S[j][e] = (v < V && kk < K) ? pool[(size_t)v * K + kk] : 0.f;
    }
  const float negA = -expf(A_log[h]), bias = dt_bias[h], q_scale = 1.f / sqrtf((float)K);
  pdl_wait();
  qkv = after_wait(qkv);
  b_raw = after_wait(b_raw);
  a_raw = after_wait(a_raw);
  auto fetch = [&](int buf, int c0) {
    const int nc = min(RC_Q, n - c0);
    const __nv_bfloat16* rows = qkv + (size_t)(t0 + c0) * ldq;
    stage_rows(rows + k_off + grp * K, ldq, nc, K, GD_KP, sm.k[buf], LK, vec);
    stage_rows(rows + q_off + grp * K, ldq, nc, K, GD_KP, sm.q[buf], LK, vec);
    stage_rows(rows + v_off + h * V + v0, ldq, nc, V - v0, GD_VS, sm.v[buf], LV, vec);
    cp_async_commit();
  };
  fetch(0, 0);
  const int ti = warp >> 1, c16 = 16 * (warp & 1);      // rows 16 ti .. of the chunk; columns c16 .. of the slice
  for (int c0 = 0, buf = 0; c0 < n; c0 += RC_Q, buf ^= 1) {
    const int nc = min(RC_Q, n - c0);
    const __nv_bfloat16 *sk = sm.k[buf], *sq = sm.q[buf], *sv = sm.v[buf];
    cp_async_wait();
    __syncthreads();      // the chunk before has been read, this one's rows are there
    delta_rows(sm, sk, sq, a_raw + (size_t)(t0 + c0) * lda + h, lda, b_raw + (size_t)(t0 + c0) * ldb + h, ldb, nc, negA, bias, q_scale);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        store_split(sm.state[0] + (16 * vi + g + (e >> 1) * 8) * LK + 16 * ni + 8 * j + 2 * q, GD_VS * LK, S[j][e], S[j][e + 1]);
    __syncthreads();
    if (c0 + RC_Q < n) fetch(buf ^ 1, c0 + RC_Q);
    unsigned ak[GD_KP / 16][4], aq[GD_KP / 16][4];      // this warp's 16 rows of k and of q
#pragma unroll
    for (int k = 0; k < GD_KP / 16; ++k) {
      frag_a(ak[k], sk + 16 * ti * LK + 16 * k, LK, lane);
      frag_a(aq[k], sq + 16 * ti * LK + 16 * k, LK, lane);
    }
    delta_scores(sm, sk, ak, aq, sm.p[0], LP, RC_Q * LP);
    // right sides, and what the state before the chunk gives to o
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    {
      float ks[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      float low_k[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, low_q[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int pl = 2; pl >= 0; --pl)
#pragma unroll
        for (int k = 0; k < GD_KP / 16; ++k) {
          unsigned bb[4];
          frag_b(bb, sm.state[pl] + c16 * LK + 16 * k, LK, lane);
          mma_plane(ks[0], low_k[0], pl, ak[k], bb[0], bb[1]);
          mma_plane(ks[1], low_k[1], pl, ak[k], bb[2], bb[3]);
          mma_plane(acc[0], low_q[0], pl, aq[k], bb[0], bb[1]);
          mma_plane(acc[1], low_q[1], pl, aq[k], bb[2], bb[3]);
        }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = 16 * ti + g + (e >> 1) * 8, c = c16 + 8 * j + 2 * q + (e & 1);
          sm.r[t * GD_VS + c] = sm.beta[t] * (to_f(sv[t * LV + c]) - sm.since[t] * sm.rk[t] * (ks[j][e] + low_k[j][e]));
          acc[j][e] = sm.since[t] * sm.rq[t] * (acc[j][e] + low_q[j][e]);
        }
    }
    __syncthreads();
    if (warp < 4 && lane < 16) {      // column `lane` of the inverse of diagonal block `warp`
      float x[16];
      const float* mb = sm.m + (16 * warp) * LM + 16 * warp;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float s = i == lane ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < i) s = fmaf(-mb[i * LM + j], x[j], s);
        x[i] = s;
        sm.inv[warp][i * LI + lane] = s;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int b = 0; b < 4; ++b) {      // a lane a column
      float rb[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) rb[j] = sm.r[(16 * b + j) * GD_VS + lane];
      // The inverse of a triangular block: row i takes the right sides up to its own and no others (which may not be finite).
      float ub[2] = {0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 w = reinterpret_cast<const float4*>(sm.inv[b] + (warp + 8) * LI)[j];
        const float m[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int e = 3; e >= 0; --e)
          if (4 * j + e < 8 || 4 * j + e - 8 <= warp) ub[1] = fmaf(m[e], rb[4 * j + e], ub[1]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float4 w = reinterpret_cast<const float4*>(sm.inv[b] + warp * LI)[j];
        const float m[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int e = 3; e >= 0; --e)
          if (4 * j + e <= warp) ub[0] = fmaf(m[e], rb[4 * j + e], ub[0]);
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 2; ++i) sm.r[(16 * b + warp + 8 * i) * GD_VS + lane] = ub[i];
      if (b == 3) break;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 16; ++j) rb[j] = sm.r[(16 * b + j) * GD_VS + lane];
      for (int t = 16 * (b + 1) + warp; t < RC_Q; t += 8) {
        const float4* w4 = reinterpret_cast<const float4*>(sm.m + t * LM + 16 * b);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 w = w4[j];
          s = fmaf(w.x, rb[4 * j], fmaf(w.y, rb[4 * j + 1], fmaf(w.z, rb[4 * j + 2], fmaf(w.w, rb[4 * j + 3], s))));
        }
        sm.r[t * GD_VS + lane] -= s;
      }
      __syncthreads();
    }
    __syncthreads();
    bool bad = false;                        // an update that is not finite
    for (int e = tid; e < RC_Q * GD_VS / 2; e += RC_THREADS) {
      const int s = e / (GD_VS / 2), c = 2 * (e - s * (GD_VS / 2));
      const float2 u = *reinterpret_cast<const float2*>(sm.r + s * GD_VS + c);
      const float w = sm.left[s] * sm.rk[s];
      store_split(sm.u[0] + s * LV + c, RC_Q * LV, u.x, u.y);
      store_split(sm.wu[0] + s * LV + c, RC_Q * LV, w * u.x, w * u.y);
      bad |= !(fabsf(u.x) < INFINITY && fabsf(u.y) < INFINITY);
    }
    bad = __syncthreads_or(bad);
    float low[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    for (int k = 0; k <= 16 * ti; k += 16) {      // both sides in three numbers: the six products that reach 24 bits
      unsigned a[3][4], bb[3][4];
#pragma unroll
      for (int pl = 0; pl < 3; ++pl) {
        frag_a(a[pl], sm.p[pl] + 16 * ti * LP + k, LP, lane);
        frag_b_t(bb[pl], sm.u[pl] + k * LV + c16, LV, lane);
      }
      if (bad && k == 16 * ti) {      // not finite: the first of an update's three numbers, beside zeros
#pragma unroll
        for (int i = 0; i < 4; ++i) drop_bad(bb[0][i]);
      }
#pragma unroll
      for (int sum = 2; sum >= 0; --sum)
#pragma unroll
        for (int pl = 0; pl <= sum; ++pl) {
          mma_plane(acc[0], low[0], sum, a[pl], bb[sum - pl][0], bb[sum - pl][1]);
          mma_plane(acc[1], low[1], sum, a[pl], bb[sum - pl][2], bb[sum - pl][3]);
        }
    }
    if (bad) add_bad(acc, sm.p[0], RC_Q * LP, LP, ti, c16, g, q, [&](int s, int c) { return sm.r[s * GD_VS + c]; });
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 16 * ti + g + (e >> 1) * 8, c = c16 + 8 * j + 2 * q + (e & 1);
        if (t < nc && v0 + c < V) o[(size_t)(t0 + c0 + t) * ldo + h * V + v0 + c] = acc[j][e] + low[j][e];
      }
    const float keep = sm.since[RC_Q - 1];
    float add[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, add_low[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int k = 0; k < RC_Q; k += 16) {
      unsigned bb[4];
      frag_b_t(bb, sk + k * LK + 16 * ni, LK, lane);
#pragma unroll
      for (int pl = 2; pl >= 0; --pl) {
        unsigned a[4];
        frag_a_t(a, sm.wu[pl] + k * LV + 16 * vi, LV, lane);
        mma_plane(add[0], add_low[0], pl, a, bb[0], bb[1]);
        mma_plane(add[1], add_low[1], pl, a, bb[2], bb[3]);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf(keep, S[j][e], add[j][e] + add_low[j][e]);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int v = v0 + 16 * vi + g + (e >> 1) * 8, kk = 16 * ni + 8 * j + 2 * q + (e & 1);
      if (v < V && kk < K) pool[(size_t)v * K + kk] = S[j][e];
    }
}

// The chain above is a chunk's phases one after the other, and most of them do not need the state.  With fewer states than SMs:
//   first pass   every chunk of every run side by side: decays, P and T = (I + M)^-1, each kept as the three numbers that the
//                products take.  T is made in 64 bits: with keys that repeat, rounding it on the way to 32 left U 1.2 times the
//                error of the solution by blocks above.  The blocks of 16 on the diagonal first, then those under it by
//                T_ij = -T_ii (M_ij T_jj + ... + M_i,i-1 T_i-1,j), one distance from the diagonal after the other
//   second pass  a block a (request, head, 32 columns) walks the run:  R = beta (v - G k . S),  U = T R,
//                o = G q . S + P U,  S = G_end S + K^T (what is left of U): three products and four barriers a chunk
// 1024 rows of 16 heads of 64 x 64, two requests: 162 us in one kernel, 106 in two (10 us a chunk of the chain, 4
// in the second pass); one of 200 rows 43 and 35, one of 100 23 and 24.
constexpr int GD_TILE = RC_Q * RC_Q;                       // a plane of T or P in scratch memory
constexpr int GD_ROWS = 4;                                 // beta, G rk, G rq, (G_end / G) rk, each RC_Q floats, then G_end
struct DeltaChunk {                                        // what the first pass leaves of a (chunk, head)
  __nv_bfloat16 t[3][GD_TILE], p[3][GD_TILE];
  float rows[GD_ROWS][RC_Q];
  float keep[4];
};

struct DeltaFirstMemory {
  static constexpr int LK = GD_KP + 8, LM = RC_Q + 2;
  __nv_bfloat16 k[RC_Q * LK], q[RC_Q * LK];
  double m[RC_Q * LM], t[RC_Q * LM], x[3][16 * 17];
  double sum[RC_Q];
  float since[RC_Q], left[RC_Q], beta[RC_Q], rk[RC_Q], rq[RC_Q];
};

__global__ void __launch_bounds__(RC_THREADS, 2)
gated_delta_first_kernel(const __nv_bfloat16* qkv, int ldq, int q_off, int k_off, const __nv_bfloat16* b_raw, int ldb,
                         const __nv_bfloat16* a_raw, int lda, const float* __restrict__ dt_bias, const float* __restrict__ A_log,
                         const int* __restrict__ token_req, const int* __restrict__ req_first_token, const int* __restrict__ requests,
                         int n_requests, ChunkRule rule, DeltaChunk* chunks, int H, int G, int K, int vec) {
  extern __shared__ __align__(16) char rc_sm[];
  DeltaFirstMemory& sm = *reinterpret_cast<DeltaFirstMemory*>(rc_sm);
  constexpr int LK = DeltaFirstMemory::LK, LM = DeltaFirstMemory::LM;
  const int h = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ti = warp >> 1, grp = h / (H / G);
  pdl_trigger();
  const ChunkJob job = find_job(req_first_token, requests, n_requests, blockIdx.y, RC_Q);
  const int t_first = job.r >= 0 ? req_first_token[job.r] : 0, t_end = job.r >= 0 ? req_first_token[job.r + 1] : 0;
  const int n = run_length(token_req, t_first, t_end, job.r);
  const float negA = -expf(A_log[h]), bias = dt_bias[h], q_scale = 1.f / sqrtf((float)K);
  pdl_wait();
  if (job.c * RC_Q >= n || !rule.chunks(n)) return;
  qkv = after_wait(qkv);
  b_raw = after_wait(b_raw);
  a_raw = after_wait(a_raw);
  chunks = after_wait(chunks);
  const int t0 = t_first + job.c * RC_Q, nc = min(RC_Q, n - job.c * RC_Q);
  stage_rows(qkv + (size_t)t0 * ldq + k_off + grp * K, ldq, nc, K, GD_KP, sm.k, LK, vec);
  stage_rows(qkv + (size_t)t0 * ldq + q_off + grp * K, ldq, nc, K, GD_KP, sm.q, LK, vec);
  cp_async_commit();
  cp_async_wait();
  __syncthreads();
  delta_rows(sm, sm.k, sm.q, a_raw + (size_t)t0 * lda + h, lda, b_raw + (size_t)t0 * ldb + h, ldb, nc, negA, bias, q_scale);
  __syncthreads();
  DeltaChunk& out = chunks[(size_t)blockIdx.y * H + h];
  {
    unsigned ak[GD_KP / 16][4], aq[GD_KP / 16][4];
#pragma unroll
    for (int k = 0; k < GD_KP / 16; ++k) {
      frag_a(ak[k], sm.k + 16 * ti * LK + 16 * k, LK, lane);
      frag_a(aq[k], sm.q + 16 * ti * LK + 16 * k, LK, lane);
    }
    delta_scores(sm, sm.k, ak, aq, out.p[0], RC_Q, GD_TILE);
  }
  if (tid < RC_Q) {
    out.rows[0][tid] = sm.beta[tid];
    out.rows[1][tid] = sm.since[tid] * sm.rk[tid];
    out.rows[2][tid] = sm.since[tid] * sm.rq[tid];
    out.rows[3][tid] = sm.left[tid] * sm.rk[tid];
    if (tid == RC_Q - 1) out.keep[0] = sm.since[tid];
  }
  __syncthreads();
  if (tid < RC_Q) {      // a column of a block on the diagonal
    const int b16 = 16 * (tid >> 4), col = tid & 15;
    double x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      double s[2] = {i == col ? 1. : 0., 0.};
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < i) s[j & 1] = fma(-sm.m[(b16 + i) * LM + b16 + j], x[j], s[j & 1]);
      x[i] = s[0] + s[1];
      sm.t[(b16 + i) * LM + b16 + col] = i < col ? 0. : x[i];      // (also where a row is not finite)
    }
  }
  __syncthreads();
  const int ra = tid >> 4, cb = tid & 15;      // a thread an element of a block
#pragma unroll 1
  for (int d = 1; d < 4; ++d) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {              // blocks (j + d, j)
      if (j + d >= 4) continue;
      double s[4] = {0., 0., 0., 0.};
      const double *m = sm.m + (16 * (j + d) + ra) * LM + 16 * j, *t = sm.t + 16 * j * LM + 16 * j + cb;
      for (int k = 0; k < 16 * d; k += 4)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = fma(m[k + e], t[(k + e) * LM], s[e]);
      sm.x[j][ra * 17 + cb] = (s[0] + s[1]) + (s[2] + s[3]);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (j + d >= 4) continue;
      double s[4] = {0., 0., 0., 0.};
      const double *w = sm.t + (16 * (j + d) + ra) * LM + 16 * (j + d), *x = sm.x[j] + cb;
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k <= ra) s[k & 3] = fma(-w[k], x[k * 17], s[k & 3]);      // (rows up to its own, and no others, which may not be finite)
      sm.t[(16 * (j + d) + ra) * LM + 16 * j + cb] = (s[0] + s[1]) + (s[2] + s[3]);
    }
    __syncthreads();
  }
  for (int e = tid; e < RC_Q * RC_Q / 2; e += RC_THREADS) {
    const int i = e >> 5, j = 2 * (e & 31);
    if (j / 16 > i / 16) continue;             // up to the diagonal's block
    __nv_bfloat162 part[3];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      double x = sm.t[i * LM + j + c];
      const bool finite = fabs(x) < 3e38;
#pragma unroll
      for (int pl = 0; pl < 3; ++pl) {         // a number that is not finite is the first of them, beside zeros
        const __nv_bfloat16 v = __float2bfloat16_rn((float)x);
        if (c == 0) part[pl].x = v; else part[pl].y = v;
        x = finite ? x - (double)__bfloat162float(v) : 0.;
      }
    }
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) *reinterpret_cast<__nv_bfloat162*>(out.t[pl] + i * RC_Q + j) = part[pl];
  }
}

struct DeltaSecondMemory {
  static constexpr int LK = GD_KP + 8, LV = GD_VS + 8, LP = RC_Q + 8;
  __nv_bfloat16 k[2][RC_Q * LK], q[2][RC_Q * LK], v[2][RC_Q * LV];
  __nv_bfloat16 t[2][3][RC_Q * LP], p[2][3][RC_Q * LP];
  __nv_bfloat16 state[3][GD_VS * LK];                                              // [column][row of the state]
  __nv_bfloat16 r[3][RC_Q * LV], u[3][RC_Q * LV], wu[3][RC_Q * LV];                // right sides, updates, what is left of them
  float rows[2][GD_ROWS + 1][RC_Q];                                                // (the last: G_end, in its first place)
};

__global__ void __launch_bounds__(RC_THREADS, 1)
gated_delta_second_kernel(const __nv_bfloat16* qkv, int ldq, int q_off, int k_off, int v_off, float* state, const int* __restrict__ slots,
                          const int* __restrict__ token_req, const int* __restrict__ req_first_token, const int* __restrict__ requests,
                          ChunkRule rule, const DeltaChunk* chunks, float* __restrict__ o, int ldo, int H, int G, int K, int V, int vec) {
  extern __shared__ __align__(16) char rc_sm[];
  DeltaSecondMemory& sm = *reinterpret_cast<DeltaSecondMemory*>(rc_sm);
  constexpr int LK = DeltaSecondMemory::LK, LV = DeltaSecondMemory::LV, LP = DeltaSecondMemory::LP;
  const int h = blockIdx.x, r = requests != nullptr ? requests[blockIdx.y] : (int)blockIdx.y, v0 = blockIdx.z * GD_VS;
  const int t0 = r >= 0 ? req_first_token[r] : 0, t1 = r >= 0 ? req_first_token[r + 1] : 0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int grp = h / (H / G);
  pdl_trigger();
  const int n = run_length(token_req, t0, t1, r);
  if (!rule.chunks(n)) {
    pdl_wait();
    return;
  }
  const int first_job = jobs_before(req_first_token, requests, blockIdx.y, RC_Q);
  // this warp's part of the state, as above
  const int vi = warp & 1, ni = warp >> 1;
  float S[2][4];
  float* pool = state + ((size_t)slots[r] * H + h) * K * V;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int v = v0 + 16 * vi + g + (e >> 1) * 8, kk = 16 * ni + 8 * j + 2 * q + (e & 1);
      S[j][e] = (v < V && kk < K) ? pool[(size_t)v * K + kk] : 0.f;
    }
  pdl_wait();
  qkv = after_wait(qkv);
  chunks = after_wait(chunks);
  auto fetch = [&](int buf, int c0) {
    const int nc = min(RC_Q, n - c0);
    const __nv_bfloat16* rows = qkv + (size_t)(t0 + c0) * ldq;
    const DeltaChunk& in = chunks[(size_t)(first_job + c0 / RC_Q) * H + h];
    stage_rows(rows + k_off + grp * K, ldq, nc, K, GD_KP, sm.k[buf], LK, vec);
    stage_rows(rows + q_off + grp * K, ldq, nc, K, GD_KP, sm.q[buf], LK, vec);
    stage_rows(rows + v_off + h * V + v0, ldq, nc, V - v0, GD_VS, sm.v[buf], LV, vec);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl)
#pragma unroll
      for (int i = 0; i < RC_Q * RC_Q / 8 / RC_THREADS; ++i) {
        const int e = tid + i * RC_THREADS, row = e >> 3, c = (e & 7) * 8;
        if (c / 16 > row / 16) continue;                  // up to the diagonal's tile
        cp_async16(sm.t[buf][pl] + row * LP + c, in.t[pl] + row * RC_Q + c, true);
        cp_async16(sm.p[buf][pl] + row * LP + c, in.p[pl] + row * RC_Q + c, true);
      }
    if (tid < GD_ROWS * RC_Q / 4) cp_async16(sm.rows[buf][0] + 4 * tid, in.rows[0] + 4 * tid, true);
    else if (tid == GD_ROWS * RC_Q / 4) cp_async16(sm.rows[buf][GD_ROWS], in.keep, true);
    cp_async_commit();
  };
  fetch(0, 0);
  const int ti = warp >> 1, c16 = 16 * (warp & 1);      // rows 16 ti .. of the chunk; columns c16 .. of the slice
  // acc += W X for this warp's rows and columns, W (lower triangular) and X in three numbers: the six products that reach 24 bits.
  // bad: X has values that are not finite (the first of their three numbers, beside zeros).
  auto times_lower = [&](float (&acc)[2][4], const __nv_bfloat16 (&w)[3][RC_Q * LP], const __nv_bfloat16 (&x)[3][RC_Q * LV], bool bad) {
    float low[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    for (int k = 0; k <= 16 * ti; k += 16) {
      unsigned a[3][4], bb[3][4];
#pragma unroll
      for (int pl = 0; pl < 3; ++pl) {
        frag_a(a[pl], w[pl] + 16 * ti * LP + k, LP, lane);
        frag_b_t(bb[pl], x[pl] + k * LV + c16, LV, lane);
      }
      if (bad && k == 16 * ti) {
#pragma unroll
        for (int i = 0; i < 4; ++i) drop_bad(bb[0][i]);
      }
#pragma unroll
      for (int sum = 2; sum >= 0; --sum)
#pragma unroll
        for (int pl = 0; pl <= sum; ++pl) {
          mma_plane(acc[0], low[0], sum, a[pl], bb[sum - pl][0], bb[sum - pl][1]);
          mma_plane(acc[1], low[1], sum, a[pl], bb[sum - pl][2], bb[sum - pl][3]);
        }
    }
    if (bad) add_bad(acc, w[0], RC_Q * LP, LP, ti, c16, g, q, [&](int s, int c) { return to_f(x[0][s * LV + c]); });
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] += low[j][e];
  };
  for (int c0 = 0, buf = 0; c0 < n; c0 += RC_Q, buf ^= 1) {
    const int nc = min(RC_Q, n - c0);
    const __nv_bfloat16 *sk = sm.k[buf], *sq = sm.q[buf], *sv = sm.v[buf];
    cp_async_wait();
#pragma unroll
    for (int j = 0; j < 2; ++j)      // (the planes of the state were last read two barriers ago)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        store_split(sm.state[0] + (16 * vi + g + (e >> 1) * 8) * LK + 16 * ni + 8 * j + 2 * q, GD_VS * LK, S[j][e], S[j][e + 1]);
    __syncthreads();      // the chunk before has been read, this one's rows and the state are there
    if (c0 + RC_Q < n) fetch(buf ^ 1, c0 + RC_Q);
    const float* rows = sm.rows[buf][0];
    // right sides, and what the state before the chunk gives to o
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    bool bad = false;
    {
      float ks[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      float low_k[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, low_q[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int k = 0; k < GD_KP / 16; ++k) {
        unsigned ak[4], aq[4];
        frag_a(ak, sk + 16 * ti * LK + 16 * k, LK, lane);
        frag_a(aq, sq + 16 * ti * LK + 16 * k, LK, lane);
#pragma unroll
        for (int pl = 2; pl >= 0; --pl) {
          unsigned bb[4];
          frag_b(bb, sm.state[pl] + c16 * LK + 16 * k, LK, lane);
          mma_plane(ks[0], low_k[0], pl, ak, bb[0], bb[1]);
          mma_plane(ks[1], low_k[1], pl, ak, bb[2], bb[3]);
          mma_plane(acc[0], low_q[0], pl, aq, bb[0], bb[1]);
          mma_plane(acc[1], low_q[1], pl, aq, bb[2], bb[3]);
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const int t = 16 * ti + g + (e >> 1) * 8, c = c16 + 8 * j + 2 * q;
          float w[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            w[i] = rows[t] * (to_f(sv[t * LV + c + i]) - rows[RC_Q + t] * (ks[j][e + i] + low_k[j][e + i]));
            bad |= !(fabsf(w[i]) < INFINITY);
            acc[j][e + i] = rows[2 * RC_Q + t] * (acc[j][e + i] + low_q[j][e + i]);
          }
          store_split(sm.r[0] + t * LV + c, RC_Q * LV, w[0], w[1]);
        }
    }
    bad = __syncthreads_or(bad);
    float u[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    times_lower(u, sm.t[buf], sm.r, bad);
    bad = false;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int t = 16 * ti + g + (e >> 1) * 8, c = c16 + 8 * j + 2 * q;
        const float w = rows[3 * RC_Q + t];
        store_split(sm.u[0] + t * LV + c, RC_Q * LV, u[j][e], u[j][e + 1]);
        store_split(sm.wu[0] + t * LV + c, RC_Q * LV, w * u[j][e], w * u[j][e + 1]);
        bad |= !(fabsf(u[j][e]) < INFINITY && fabsf(u[j][e + 1]) < INFINITY);
      }
    bad = __syncthreads_or(bad);
    const float keep = sm.rows[buf][GD_ROWS][0];
    float add[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, add_low[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int k = 0; k < RC_Q; k += 16) {
      unsigned bb[4];
      frag_b_t(bb, sk + k * LK + 16 * ni, LK, lane);
#pragma unroll
      for (int pl = 2; pl >= 0; --pl) {
        unsigned a[4];
        frag_a_t(a, sm.wu[pl] + k * LV + 16 * vi, LV, lane);
        mma_plane(add[0], add_low[0], pl, a, bb[0], bb[1]);
        mma_plane(add[1], add_low[1], pl, a, bb[2], bb[3]);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf(keep, S[j][e], add[j][e] + add_low[j][e]);
    times_lower(acc, sm.p[buf], sm.u, bad);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 16 * ti + g + (e >> 1) * 8, c = c16 + 8 * j + 2 * q + (e & 1);
        if (t < nc && v0 + c < V) o[(size_t)(t0 + c0 + t) * ldo + h * V + v0 + c] = acc[j][e];
      }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int v = v0 + 16 * vi + g + (e >> 1) * 8, kk = 16 * ni + 8 * j + 2 * q + (e & 1);
      if (v < V && kk < K) pool[(size_t)v * K + kk] = S[j][e];
    }
}

// Floats of scratch memory for the two passes over runs of `jobs` chunks at most.
MLXB_EXPORT long long mlxb_gated_delta_chunks_scratch(int jobs, int H) {
  return (long long)jobs * H * (long long)(sizeof(DeltaChunk) / sizeof(float));
}

// The arguments of mlxb_gated_delta_scan (bfloat16 inputs, states of up to 64 rows); requests with a single row are left out.
// scratch: null (one kernel), or memory of mlxb_gated_delta_chunks_scratch floats, 16-byte aligned (two passes).  jobs: the chunks of
// the listed requests' rows, no fewer (their rows / 64 and a chunk a request are enough).
MLXB_EXPORT int mlxb_gated_delta_chunks(const void* qkv, int ldq, int q_off, int k_off, int v_off, const void* b_raw, int ldb,
                                        const void* a_raw, int lda, const float* dt_bias, const float* A_log, float* state,
                                        const int* slots, const int* token_req, const int* req_first_token, float* o, int ldo, int H,
                                        int G, int K, int V, const int* requests, int n_requests, int scan_fixed, int scan_row,
                                        int chunk_fixed, int chunk_each, int jobs, float* scratch, cudaStream_t stream) {
  if (n_requests <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || K <= 0 || V <= 0 || K > GD_KP || n_requests > 65535)
    return mlxb_fail(MLXB_BAD_ARG, "gated_delta_chunks: %d heads over %d key heads, state %d x %d (at most %d rows)", H, G, K, V, GD_KP);
  const int vec = (((uintptr_t)qkv & 15) == 0 && ldq % 8 == 0 && q_off % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0 && K % 8 == 0 &&
                   V % 8 == 0);
  if (scratch != nullptr) {
    if (jobs <= 0 || jobs > 65535 || ((uintptr_t)scratch & 15))
      return mlxb_fail(MLXB_BAD_ARG, "gated_delta_chunks: %d chunks of %d requests, scratch memory 16-byte aligned", jobs, n_requests);
    static_assert(sizeof(DeltaChunk) % 16 == 0 && sizeof(DeltaSecondMemory) <= 227 * 1024, "pieces of 16 bytes; a block's shared memory");
    static SharedLimit limits[2];
    cudaError_t e = limits[0].raise(gated_delta_first_kernel, sizeof(DeltaFirstMemory));
    if (e == cudaSuccess) e = limits[1].raise(gated_delta_second_kernel, sizeof(DeltaSecondMemory));
    if (e != cudaSuccess) return mlxb_fail((int)e, "gated_delta_chunks: %zu bytes of shared memory: %s", sizeof(DeltaSecondMemory), cudaGetErrorString(e));
    const ChunkRule rule = {scan_fixed, scan_row, chunk_fixed, chunk_each};
    launch_pdl(gated_delta_first_kernel, dim3(H, (unsigned)jobs), dim3(RC_THREADS), sizeof(DeltaFirstMemory), stream,
               (const __nv_bfloat16*)qkv, ldq, q_off, k_off, (const __nv_bfloat16*)b_raw, ldb, (const __nv_bfloat16*)a_raw, lda, dt_bias,
               A_log, token_req, req_first_token, requests, n_requests, rule, (DeltaChunk*)scratch, H, G, K, vec);
    if (int err = mlxb_check_launch("gated_delta_chunks (first pass)")) return err;
    launch_pdl(gated_delta_second_kernel, dim3(H, n_requests, (V + GD_VS - 1) / GD_VS), dim3(RC_THREADS), sizeof(DeltaSecondMemory), stream,
               (const __nv_bfloat16*)qkv, ldq, q_off, k_off, v_off, state, slots, token_req, req_first_token, requests, rule,
               (const DeltaChunk*)scratch, o, ldo, H, G, K, V, vec);
    return mlxb_check_launch("gated_delta_chunks (second pass)");
  }
  const size_t smem = sizeof(DeltaMemory);
  static SharedLimit limit;
  const cudaError_t e = limit.raise(gated_delta_chunks_kernel, smem);
  if (e != cudaSuccess) return mlxb_fail((int)e, "gated_delta_chunks: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  launch_pdl(gated_delta_chunks_kernel, dim3(H, n_requests, (V + GD_VS - 1) / GD_VS), dim3(RC_THREADS), smem, stream,
             (const __nv_bfloat16*)qkv, ldq, q_off, k_off, v_off, (const __nv_bfloat16*)b_raw, ldb, (const __nv_bfloat16*)a_raw, lda,
             dt_bias, A_log, state, slots, token_req, req_first_token, requests, ChunkRule{scan_fixed, scan_row, chunk_fixed, chunk_each}, o, ldo,
             H, G, K, V, vec);
  return mlxb_check_launch("gated_delta_chunks");
}
