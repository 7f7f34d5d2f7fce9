// Time mixing in the manner of RWKV: a linear recurrence per head whose decay is computed from the data, read
// through mixes of every token with the token before it.
//
// token_shift_mix      out[t, s*sec + c] = x[t, c] + (prev[t, c] - x[t, c]) * mu[s, c] for each of n_mix mixes s, where
//                      prev is the row before t of the same request: a row of this step, or, for the request's
//                      first row of the step, the last row of the step before, kept in the state (zeros at position 0).
// shift_state_update   moves the last row of every request's run into the state (launched after the mix).
// wkv_scan             per (request, head), state S of K rows (key channels) and V columns, float32:
//                        o_t[v] = sum_k r_t[k] (S[k, v] + u[k] k_t[k] v_t[v])      (the bonus u for the current token only)
//                        S[k, v] <- w_t[k] S[k, v] + k_t[k] v_t[v],   w_t[k] = exp(-exp(d_t[k]))
//                      d_t arrives in float32 (the decay's projection with its bias); exponentials, state and sums
//                      are float32; r, k, v arrive in the activation dtype.
//
// A request's rows of a step are req_first_token[r] .. (as many as carry its index in token_req); its state lives
// in row slots[r] of a float32 pool ([slots, H, V, K]: a head's state column by column), read at the start of the
// run and written back at its end.  A thread holds 16 consecutive rows of one column in registers; the NS threads of
// a column are neighbouring lanes and add their partial sums by shuffles; 16 tokens at a time are staged in shared
// memory.  Token by token the order of additions for a token depends on the layer's sizes only; in chunks (wkv_chunks below, which
// the engine's sizes take) also on where its run begins, that is on how a prompt was cut into steps, in float32 as in bfloat16.
#include <type_traits>

#include "common.cuh"
#include "recurrent_tiles.cuh"

MLXB_DEFINE_LAST_ERROR()

template <typename T>
__global__ void token_shift_mix_kernel(const T* x, int ldx, const float* __restrict__ mu, int n_mix, int D,
                                       const float* state, const int* __restrict__ slots,
                                       const int* __restrict__ positions, const int* __restrict__ token_req,
                                       const int* __restrict__ req_first_token, T* __restrict__ out, int ldo, int sec) {
  const int t = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = token_req[t];
  if (r < 0 || c >= D) return;
  pdl_wait();
  pdl_trigger();
  x = after_wait(x);
  state = after_wait(state);
  const float cur = to_f(x[(size_t)t * ldx + c]);
  float prev;
  if (t > req_first_token[r]) prev = to_f(x[(size_t)(t - 1) * ldx + c]);
  else prev = positions[t] > 0 ? state[(size_t)slots[r] * D + c] : 0.f;
  const float diff = prev - cur;
  for (int s = 0; s < n_mix; ++s)
    out[(size_t)t * ldo + (size_t)s * sec + c] = from_f<T>(fmaf(diff, mu[(size_t)s * D + c], cur));
}

template <typename T>
__global__ void shift_state_update_kernel(const T* x, int ldx, int D, float* state, const int* __restrict__ slots,
                                          const int* __restrict__ token_req, const int* __restrict__ req_first_token) {
  pdl_wait();
  pdl_trigger();
  x = after_wait(x);
  const int r = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
  const int t0 = req_first_token[r], t1 = req_first_token[r + 1];
  const int n = run_length(token_req, t0, t1, r);
  if (n == 0 || c >= D) return;
  state[(size_t)slots[r] * D + c] = to_f(x[(size_t)(t0 + n - 1) * ldx + c]);
}

// x: [n_tokens, >= D] (activation dtype); mu: float32 [n_mix, D]; state: float32 [slots, D]; out: [n_tokens, n_mix*sec],
// mix s in columns s*sec .. s*sec + D - 1 (sec >= D).
MLXB_EXPORT int mlxb_token_shift_mix(int dtype, const void* x, int ldx, const float* mu, int n_mix, int D, float* state,
                                     const int* slots, const int* positions, const int* token_req,
                                     const int* req_first_token, void* out, int ldo, int sec, int n_tokens, int n_requests,
                                     cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (D <= 0 || n_mix <= 0 || ldx < D || sec < D || ldo < n_mix * sec || n_tokens > 65535 * 32 || n_requests > 65535)
    return mlxb_fail(MLXB_BAD_ARG, "token_shift_mix: %d mixes of width %d, strides %d / %d", n_mix, D, ldx, ldo);
  const int threads = D >= 256 ? 256 : 128;
  const dim3 grid((D + threads - 1) / threads, n_tokens), sgrid((D + threads - 1) / threads, n_requests);
  if (dtype == MLXB_F32) {
    launch_pdl(token_shift_mix_kernel<float>, grid, dim3(threads), 0, stream, (const float*)x, ldx, mu, n_mix, D,
               (const float*)state, slots, positions, token_req, req_first_token, (float*)out, ldo, sec);
    if (int e = mlxb_check_launch("token_shift_mix")) return e;
    launch_pdl(shift_state_update_kernel<float>, sgrid, dim3(threads), 0, stream, (const float*)x, ldx, D, state, slots,
               token_req, req_first_token);
  } else if (dtype == MLXB_BF16) {
    launch_pdl(token_shift_mix_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream, (const __nv_bfloat16*)x, ldx, mu,
               n_mix, D, (const float*)state, slots, positions, token_req, req_first_token, (__nv_bfloat16*)out, ldo, sec);
    if (int e = mlxb_check_launch("token_shift_mix")) return e;
    launch_pdl(shift_state_update_kernel<__nv_bfloat16>, sgrid, dim3(threads), 0, stream, (const __nv_bfloat16*)x, ldx, D,
               state, slots, token_req, req_first_token);
  } else {
    return mlxb_fail(MLXB_BAD_DTYPE, "token_shift_mix: dtype code %d", dtype);
  }
  return mlxb_check_launch("shift_state_update");
}

// ---------------------------------------------------------------- the recurrence

constexpr int WK_NPT = 16;     // rows of a state column a thread holds
constexpr int WK_SEG = 20;     // floats between the staged runs of 16 rows (keeps 16-byte loads of neighbouring lanes apart)
constexpr int WK_CHUNK = 16;   // tokens staged at a time

template <typename T, int NS>
__global__ void __launch_bounds__(256)
wkv_scan_kernel(const T* rkv, int ld, int r_off, int k_off, int v_off, const float* d_raw, int ldd,
                const float* __restrict__ u, float* state, const int* __restrict__ slots,
                const int* __restrict__ token_req, const int* __restrict__ req_first_token, float* __restrict__ o,
                int ldo, int H, int K, int V, int VB) {
  extern __shared__ __align__(16) float wk_sm[];
  constexpr int NP = NS * WK_SEG;
  float* sr = wk_sm;                       // [CHUNK][NP]
  float* sk = sr + WK_CHUNK * NP;          // [CHUNK][NP]
  float* sw = sk + WK_CHUNK * NP;          // [CHUNK][NP]
  float* sv = sw + WK_CHUNK * NP;          // [CHUNK][VB]
  float* sb = sv + WK_CHUNK * VB;          // [CHUNK] sum_k r u k of the token
  const int h = blockIdx.x, r = blockIdx.y, vb = blockIdx.z;
  const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nthreads >> 5;
  const int s = tid % NS, vl = tid / NS, v = vb * VB + vl;
  const bool valid = v < V;
  pdl_wait();
  pdl_trigger();
  rkv = after_wait(rkv);
  d_raw = after_wait(d_raw);
  state = after_wait(state);
  const int t0 = req_first_token[r], t1 = req_first_token[r + 1];
  const int n = run_length(token_req, t0, t1, r);
  if (n == 0) return;
  float* st = state + (((size_t)slots[r] * H + h) * V + (valid ? v : 0)) * K;   // this thread's column
  float S[WK_NPT];
#pragma unroll
  for (int i = 0; i < WK_NPT; ++i) {
    const int kk = s * WK_NPT + i;
    S[i] = (valid && kk < K) ? st[kk] : 0.f;
  }
  for (int e = tid; e < 3 * WK_CHUNK * NP; e += nthreads) sr[e] = 0.f;     // rows beyond K stay zero
  const float* uh = u + (size_t)h * K;
  // the staged tokens of a chunk through the recurrence
  auto run_tokens = [&](int c0, int nc) {
#pragma unroll 4
    for (int tok = 0; tok < nc; ++tok) {
      const float* pr = sr + tok * NP + s * WK_SEG;
      const float* pk = sk + tok * NP + s * WK_SEG;
      const float* pw = sw + tok * NP + s * WK_SEG;
      const float vv = sv[tok * VB + vl];
      float a = 0.f;
#pragma unroll
      for (int i = 0; i < WK_NPT; i += 4) {
        const float4 r4 = *reinterpret_cast<const float4*>(pr + i);
        const float4 k4 = *reinterpret_cast<const float4*>(pk + i);
        const float4 w4 = *reinterpret_cast<const float4*>(pw + i);
        a = fmaf(r4.x, S[i], a);
        a = fmaf(r4.y, S[i + 1], a);
        a = fmaf(r4.z, S[i + 2], a);
        a = fmaf(r4.w, S[i + 3], a);
        S[i] = fmaf(w4.x, S[i], k4.x * vv);
        S[i + 1] = fmaf(w4.y, S[i + 1], k4.y * vv);
        S[i + 2] = fmaf(w4.z, S[i + 2], k4.z * vv);
        S[i + 3] = fmaf(w4.w, S[i + 3], k4.w * vv);
      }
#pragma unroll
      for (int off = NS / 2; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
      if (s == 0 && valid) o[(size_t)(t0 + c0 + tok) * ldo + h * V + v] = fmaf(sb[tok], vv, a);
    }
  };
  for (int c0 = 0; c0 < n; c0 += WK_CHUNK) {
    const int nc = min(WK_CHUNK, n - c0);
    __syncthreads();
    for (int e = tid; e < nc * K; e += nthreads) {
      const int tok = e / K, kk = e - tok * K;
      const size_t row = (size_t)(t0 + c0 + tok);
      const int at = tok * NP + (kk / WK_NPT) * WK_SEG + (kk % WK_NPT);
      sr[at] = to_f(rkv[row * ld + r_off + h * K + kk]);
      sk[at] = to_f(rkv[row * ld + k_off + h * K + kk]);
      sw[at] = expf(-expf(d_raw[row * ldd + h * K + kk]));
    }
    for (int e = tid; e < nc * VB; e += nthreads) {
      const int tok = e / VB, c = e - tok * VB;
      sv[e] = vb * VB + c < V ? to_f(rkv[(size_t)(t0 + c0 + tok) * ld + v_off + h * V + vb * VB + c]) : 0.f;
    }
    __syncthreads();
    for (int tok = warp; tok < nc; tok += nwarps) {
      float b = 0.f;
      for (int kk = lane; kk < K; kk += 32) {
        const int at = tok * NP + (kk / WK_NPT) * WK_SEG + (kk % WK_NPT);
        b = fmaf(sr[at] * uh[kk], sk[at], b);
      }
      b = warp_sum(b);
      if (lane == 0) sb[tok] = b;
    }
    __syncthreads();
    run_tokens(c0, nc);
  }
  if (valid) {
#pragma unroll
    for (int i = 0; i < WK_NPT; ++i) {
      const int kk = s * WK_NPT + i;
      if (kk < K) st[kk] = S[i];
    }
  }
}

// ---------------------------------------------------------------- the recurrence in chunks

// Token by token a run is a chain as long as it is, on as many SMs as there are (request, head) pairs: 731, 683 and 613 rows of 16
// heads of 64 took 217 us with the next tokens fetched ahead (474 without, as the scan above is), in chunks 90; a decode step of 8
// requests 9.2 and 7.0.  The state is linear in the state before, channel by channel: over a chunk of rows, S_end = W S_0 + L with W
// the product of the chunk's decays (one number a key channel) and L the state that the chunk leaves of an empty one.  So the
// chunks of a run are walked side by side:
//   first pass   chunk 0 of a run as a scan, with its outputs; of every other chunk but the last L and W
//   second pass  every chunk after the first: its state from the chunks before, then the scan with its outputs
// in float32 like the scan, in the same order within a chunk.  What bounds it then is the loads of r, k, w from shared memory that feed
// the FMAs (shared memory busy in 35 and 39 % of the cycles, ten warps an SM), so a thread has two columns (32
// numbers of the state) and multiplies pairs of channels (fma.rn.f32x2).
constexpr int WC_Q = 64;       // rows of a chunk
constexpr int WC_VB = 64;      // columns of a block: NS threads for every two of them

typedef unsigned long long f32x2;      // two float32, the first in the low half
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 twice(float v) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}
__device__ __forceinline__ float sum2(f32x2 v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); }

template <int NS>
struct WkvMemory {
  static constexpr int NP = NS * WK_SEG;
  float r[WK_CHUNK][NP], k[WK_CHUNK][NP], w[WK_CHUNK][NP];
  float v[WK_CHUNK][WC_VB];
  float bonus[WK_CHUNK];      // sum_k r u k of the token
};

// kept: [chunks before last ones][H][V][K] states (the first pass leaves the state after a run's first chunk, L of the others; then the
// state after each), then [..][H][K] products W.
template <typename T, int NS, bool FIRST>
__global__ void __launch_bounds__(32 * NS)
wkv_chunks_kernel(const T* rkv, int ld, int r_off, int k_off, int v_off, const float* d_raw, int ldd, const float* __restrict__ u,
                  float* state, const int* __restrict__ slots, const int* __restrict__ token_req,
                  const int* __restrict__ req_first_token, int n_requests, float* o, int ldo, int H, int V, float* kept,
                  float* products, bool states_ready) {
  extern __shared__ __align__(16) char wc_sm[];
  WkvMemory<NS>* sm = reinterpret_cast<WkvMemory<NS>*>(wc_sm);      // two: the next tokens are staged beside these
  constexpr int K = NS * WK_NPT, THREADS = 32 * NS, PER_TOK = K / 8;
  const int h = blockIdx.x, v0 = blockIdx.z * WC_VB, tid = threadIdx.x;
  const int s = tid % NS, col = 2 * (tid / NS);      // rows 16 s .. of columns col, col + 1 of the slice
  const bool valid = v0 + col < V;                   // (V is even)
  pdl_trigger();
  const ChunkJob job = find_job(req_first_token, nullptr, n_requests, blockIdx.y, WC_Q);
  const int t_first = job.r >= 0 ? req_first_token[job.r] : 0, t_end = job.r >= 0 ? req_first_token[job.r + 1] : 0;
  const int n = run_length(token_req, t_first, t_end, job.r);
  const bool last = (job.c + 1) * WC_Q >= n;
  pdl_wait();
  if (job.c * WC_Q >= n || (FIRST ? job.c > 0 && last : job.c == 0)) return;
  rkv = after_wait(rkv);
  d_raw = after_wait(d_raw);
  state = after_wait(state);
  kept = after_wait(kept);
  products = after_wait(products);
  const bool outputs = !FIRST || job.c == 0;
  const int t0 = t_first + job.c * WC_Q, rows = min(WC_Q, n - job.c * WC_Q);
  const size_t at = ((size_t)h * V + (valid ? v0 + col : 0)) * K + s * WK_NPT;      // of this thread's first column in a state
  const size_t state_size = (size_t)H * V * K;
  float* pool = state + (size_t)slots[job.r] * state_size + at;
  f32x2 S[2][8];
  auto load_state = [&](const float* p) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 x = valid ? *reinterpret_cast<const ulonglong2*>(p + (size_t)c * K + 4 * i) : make_ulonglong2(0ull, 0ull);
        S[c][2 * i] = x.x;
        S[c][2 * i + 1] = x.y;
      }
  };
  auto store_state = [&](float* p) {
    if (!valid) return;
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<ulonglong2*>(p + (size_t)c * K + 4 * i) = make_ulonglong2(S[c][2 * i], S[c][2 * i + 1]);
  };
  // ---- staging: a thread eight key channels of one token; 16-byte pieces of the values
  const int tok_s = tid / PER_TOK, kk_s = (tid % PER_TOK) * 8;
  constexpr int V_PIECES = WK_CHUNK * WC_VB / 8, VP = (V_PIECES + THREADS - 1) / THREADS, WORDS = sizeof(T) / 2;
  float uv[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) uv[i] = u[(size_t)h * K + kk_s + i];
  uint4 nr[WORDS], nk[WORDS], nv[VP][WORDS];
  float4 nd[2];
  const bool vec_v = (V & 7) == 0;
  auto fetch = [&](int c0) {
    const int nc = rows - c0;
    if (tok_s < nc) {
      const size_t row = (size_t)(t0 + c0 + tok_s);
      const uint4* kp = reinterpret_cast<const uint4*>(rkv + row * ld + k_off + h * K + kk_s);
      const uint4* rp = reinterpret_cast<const uint4*>(rkv + row * ld + r_off + h * K + kk_s);
      const float4* dp = reinterpret_cast<const float4*>(d_raw + row * ldd + h * K + kk_s);
#pragma unroll
      for (int i = 0; i < WORDS; ++i) {
        nk[i] = kp[i];
        if (outputs) nr[i] = rp[i];
      }
      nd[0] = dp[0];
      nd[1] = dp[1];
    }
#pragma unroll
    for (int i = 0; i < VP; ++i) {
      const int e = tid + i * THREADS, tok = e / (WC_VB / 8), c = v0 + (e % (WC_VB / 8)) * 8;
#pragma unroll
      for (int j = 0; j < WORDS; ++j) nv[i][j] = make_uint4(0u, 0u, 0u, 0u);
      if (e >= V_PIECES || tok >= nc || c >= V) continue;
      const T* vp = rkv + (size_t)(t0 + c0 + tok) * ld + v_off + h * V + c;
      if (vec_v) {
#pragma unroll
        for (int j = 0; j < WORDS; ++j) nv[i][j] = reinterpret_cast<const uint4*>(vp)[j];
      } else {
        T* d = reinterpret_cast<T*>(nv[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (c + j < V) d[j] = vp[j];
      }
    }
  };
  auto values = [](const uint4 (&raw)[WORDS], float (&f)[8]) {
    if (sizeof(T) == 2) {
      unpack8(raw[0], f);
    } else {
      *reinterpret_cast<uint4*>(f) = raw[0];
      *reinterpret_cast<uint4*>(f + 4) = raw[WORDS - 1];
    }
  };
  auto stage = [&](WkvMemory<NS>& m, int c0) {
    const bool have = tok_s < rows - c0;      // a row beyond the run changes nothing: no decay, nothing added
    float kv[8], rv[8], b = 0.f;
    values(nk, kv);
    values(nr, rv);
    const float dv[8] = {nd[0].x, nd[0].y, nd[0].z, nd[0].w, nd[1].x, nd[1].y, nd[1].z, nd[1].w};
    const int p = (kk_s / WK_NPT) * WK_SEG + (kk_s % WK_NPT);
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (!have) kv[i] = 0.f;
      if (!have || !outputs) rv[i] = 0.f;
      w[i] = have ? expf(-expf(dv[i])) : 1.f;
      b = fmaf(rv[i] * uv[i], kv[i], b);
    }
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      *reinterpret_cast<float4*>(&m.k[tok_s][p + i]) = make_float4(kv[i], kv[i + 1], kv[i + 2], kv[i + 3]);
      *reinterpret_cast<float4*>(&m.w[tok_s][p + i]) = make_float4(w[i], w[i + 1], w[i + 2], w[i + 3]);
      if (outputs) *reinterpret_cast<float4*>(&m.r[tok_s][p + i]) = make_float4(rv[i], rv[i + 1], rv[i + 2], rv[i + 3]);
    }
#pragma unroll
    for (int off = PER_TOK >> 1; off > 0; off >>= 1) b += __shfl_xor_sync(0xffffffffu, b, off);
    if (kk_s == 0) m.bonus[tok_s] = b;
#pragma unroll
    for (int i = 0; i < VP; ++i) {
      const int e = tid + i * THREADS;
      if (e >= V_PIECES) continue;
      float f[8];
      values(nv[i], f);
      float4* d = reinterpret_cast<float4*>(&m.v[e / (WC_VB / 8)][(e % (WC_VB / 8)) * 8]);
      d[0] = make_float4(f[0], f[1], f[2], f[3]);
      d[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
  };
  fetch(0);
  f32x2 prod[8];      // W, by the threads of the first columns
#pragma unroll
  for (int i = 0; i < 8; ++i) prod[i] = twice(1.f);
  if (FIRST && job.c > 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) S[0][i] = S[1][i] = 0ull;
  } else if (FIRST) {
    load_state(pool);
  } else {            // the run's state after its first chunk (or, with states_ready, after the one before), then through the chunks up to this one
    const int from = states_ready ? job.c - 1 : 0;
    const float* L = kept + (size_t)(job.base + from) * state_size + at;
    const float* W = products + ((size_t)(job.base + from) * H + h) * K + s * WK_NPT;
    load_state(L);
    for (int c = from + 1; c < job.c; ++c) {
      L += state_size;
      W += (size_t)H * K;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(W + 4 * i);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const ulonglong2 x = valid ? *reinterpret_cast<const ulonglong2*>(L + (size_t)j * K + 4 * i) : make_ulonglong2(0ull, 0ull);
          S[j][2 * i] = fma2(w.x, S[j][2 * i], x.x);
          S[j][2 * i + 1] = fma2(w.y, S[j][2 * i + 1], x.y);
        }
      }
    }
  }
  for (int c0 = 0, b = 0; c0 < rows; c0 += WK_CHUNK, b ^= 1) {
    WkvMemory<NS>& m = sm[b];
    stage(m, c0);
    __syncthreads();      // (with two buffers one barrier: the tokens before last have been read)
    if (c0 + WK_CHUNK < rows) fetch(c0 + WK_CHUNK);
    const int nc = min(WK_CHUNK, rows - c0);
#pragma unroll 1
    for (int q = 0; q < nc; q += 4) {
      float x[4][2];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 v = *reinterpret_cast<const float2*>(&m.v[q + e][col]);
        const f32x2 vv[2] = {twice(v.x), twice(v.y)};
        f32x2 acc[2] = {0ull, 0ull};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(&m.k[q + e][s * WK_SEG + 4 * i]);
          const ulonglong2 w2 = *reinterpret_cast<const ulonglong2*>(&m.w[q + e][s * WK_SEG + 4 * i]);
          if (outputs) {
            const ulonglong2 r2 = *reinterpret_cast<const ulonglong2*>(&m.r[q + e][s * WK_SEG + 4 * i]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              acc[j] = fma2(r2.x, S[j][2 * i], acc[j]);
              acc[j] = fma2(r2.y, S[j][2 * i + 1], acc[j]);
            }
          } else if (tid < NS) {
            prod[2 * i] = mul2(prod[2 * i], w2.x);
            prod[2 * i + 1] = mul2(prod[2 * i + 1], w2.y);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            S[j][2 * i] = fma2(w2.x, S[j][2 * i], mul2(k2.x, vv[j]));
            S[j][2 * i + 1] = fma2(w2.y, S[j][2 * i + 1], mul2(k2.y, vv[j]));
          }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) x[e][j] = sum2(acc[j]);
      }
      if (!outputs) continue;
      // The NS threads of a column add up: four tokens by two columns halved twice, so that a thread ends with one token
      // (NS of 1 or 2: with four or two).
      constexpr int HAVE = NS >= 4 ? 1 : NS == 2 ? 2 : 4;
      int first = 0;
      if (NS >= 2) {
        const bool up = s & 1;
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float give = up ? x[e][j] : x[e + 2][j], keep = up ? x[e + 2][j] : x[e][j];
            x[e][j] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
          }
        first = up ? 2 : 0;
      }
      if (NS >= 4) {
        const bool up = s & 2;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float give = up ? x[0][j] : x[1][j], keep = up ? x[1][j] : x[0][j];
          x[0][j] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
        }
        first += up ? 1 : 0;
      }
#pragma unroll
      for (int off = 4; off < NS; off <<= 1)
#pragma unroll
        for (int j = 0; j < 2; ++j) x[0][j] += __shfl_xor_sync(0xffffffffu, x[0][j], off);
#pragma unroll
      for (int e = 0; e < HAVE; ++e) {
        const int tok = q + first + e;
        if (s < 4 && valid && tok < nc) {
          const float2 v = *reinterpret_cast<const float2*>(&m.v[tok][col]);
          *reinterpret_cast<float2*>(o + (size_t)(t0 + c0 + tok) * ldo + h * V + v0 + col) =
              make_float2(fmaf(m.bonus[tok], v.x, x[e][0]), fmaf(m.bonus[tok], v.y, x[e][1]));
        }
      }
    }
  }
  if (last) {
    store_state(pool);
  } else if (FIRST) {
    store_state(kept + (size_t)(job.base + job.c) * state_size + at);
    if (job.c > 0 && tid < NS && blockIdx.z == 0) {
      float* W = products + ((size_t)(job.base + job.c) * H + h) * K + s * WK_NPT;
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<ulonglong2*>(W + 4 * i) = make_ulonglong2(prod[2 * i], prod[2 * i + 1]);
    }
  }
}

// Between the passes, in steps with long runs: the state after every chunk of a run in place of what the first pass left of it, so that
// the second pass does not walk through all of a run's chunks for each of them (as many reads as chunks squared).  A block has 1024
// numbers of a (request, head); the same arithmetic in the same order.  16 heads of 64, one run of 2048 rows 107 us without and 86 with
// it, of 8192 622 and 311, of 131072 97 and 15 ms; one of 512 rows 55 and 64, eight of 200 60 and 74.
constexpr int WC_LONG = 4096;  // rows of a step from which it pays: the launch takes up to 14 us, a run of as many rows gains more
constexpr int WS_AHEAD = 8;    // chunks that are asked for together
__global__ void __launch_bounds__(256)
wkv_states_kernel(const int* __restrict__ token_req, const int* __restrict__ req_first_token, float* kept, const float* products, int H,
                  int V, int K) {
  const int h = blockIdx.x, r = blockIdx.y, lane = threadIdx.x & 31;
  pdl_trigger();
  const int n = run_length(token_req, req_first_token[r], req_first_token[r + 1], r);
  int base = 0;      // kept states of the requests before
  for (int i = lane; i < r; i += 32) {
    const int len = req_first_token[i + 1] - req_first_token[i];
    base += len > WC_Q ? (len - 1) / WC_Q : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
  const int at = (blockIdx.z * 256 + threadIdx.x) * 4, size = V * K, last = (n - 1) / WC_Q;      // chunks 0 .. last - 1 are kept
  pdl_wait();
  if (at >= size || last < 2) return;
  kept = after_wait(kept);
  products = after_wait(products);
  float* L = kept + ((size_t)base * H + h) * size + at;
  const float* W = products + ((size_t)base * H + h) * K + at % K;
  const size_t next = (size_t)H * size, next_w = (size_t)H * K;
  float4 S = *reinterpret_cast<const float4*>(L);
  for (int c = 1; c < last; c += WS_AHEAD) {
    float4 l[WS_AHEAD], w[WS_AHEAD];
#pragma unroll
    for (int i = 0; i < WS_AHEAD; ++i) {
      if (c + i >= last) continue;
      l[i] = *reinterpret_cast<const float4*>(L + (size_t)(c + i) * next);
      w[i] = *reinterpret_cast<const float4*>(W + (size_t)(c + i) * next_w);
    }
#pragma unroll
    for (int i = 0; i < WS_AHEAD; ++i) {
      if (c + i >= last) continue;
      S = make_float4(fmaf(w[i].x, S.x, l[i].x), fmaf(w[i].y, S.y, l[i].y), fmaf(w[i].z, S.z, l[i].z), fmaf(w[i].w, S.w, l[i].w));
      *reinterpret_cast<float4*>(L + (size_t)(c + i) * next) = S;
    }
  }
}

// Floats of scratch memory for mlxb_wkv_chunks: states and products of the chunks before a run's last one, about as much as the step's
// outputs in float32 (V + 1 floats a key channel for every 64 rows).
MLXB_EXPORT long long mlxb_wkv_chunks_scratch(int long_rows, int H, int K, int V) {
  return (long long)(long_rows / WC_Q) * H * K * (V + 1);
}

// What the kernels take: states of 16, 32, ... 256 rows and an even number of columns, 16-byte rows of r, k and the decay.
static bool chunks_take(const void* rkv, int size, int ld, int r_off, int k_off, int v_off, const void* d_raw, int ldd, const void* state,
                        const void* o, int ldo, int K, int V) {
  const int unit = 16 / size;
  return K >= 16 && K <= 256 && (K & (K - 1)) == 0 && V % 2 == 0 && ld % unit == 0 && r_off % unit == 0 && k_off % unit == 0 &&
         (V % 8 != 0 || v_off % unit == 0) && ldd % 4 == 0 && ldo % 2 == 0 && (((uintptr_t)rkv | (uintptr_t)d_raw | (uintptr_t)state) & 15) == 0 &&
         ((uintptr_t)o & 7) == 0;
}

MLXB_EXPORT int mlxb_wkv_scan(int dtype, const void* rkv, int ld, int r_off, int k_off, int v_off, const float* d_raw,
                              int ldd, const float* u, float* state, const int* slots, const int* token_req,
                              const int* req_first_token, float* o, int ldo, int H, int K, int V, int n_requests,
                              cudaStream_t stream);

// The arguments of mlxb_wkv_scan, and scratch memory of mlxb_wkv_chunks_scratch floats (16-byte aligned).  long_rows: at least the rows
// of the step beyond the first of every request.  Sizes that the kernels do not take, and more chunks than a grid has, go token by token.
MLXB_EXPORT int mlxb_wkv_chunks(int dtype, const void* rkv, int ld, int r_off, int k_off, int v_off, const float* d_raw, int ldd,
                                const float* u, float* state, const int* slots, const int* token_req, const int* req_first_token,
                                float* o, int ldo, int H, int K, int V, int n_requests, int long_rows, float* scratch,
                                cudaStream_t stream) {
  if (n_requests <= 0 || long_rows < 0) return 0;
  const int size = dtype == MLXB_F32 ? 4 : 2;
  const long long jobs = (long long)long_rows / WC_Q + n_requests;
  if (!chunks_take(rkv, size, ld, r_off, k_off, v_off, d_raw, ldd, state, o, ldo, K, V) || ((uintptr_t)scratch & 15) || H <= 0 ||
      jobs > 65535 || (long long)V * K > 65535 * 1024LL)
    return mlxb_wkv_scan(dtype, rkv, ld, r_off, k_off, v_off, d_raw, ldd, u, state, slots, token_req, req_first_token, o, ldo, H, K, V,
                         n_requests, stream);
  float* products = scratch + (size_t)(long_rows / WC_Q) * H * V * K;
  const dim3 grid(H, (unsigned)jobs, (V + WC_VB - 1) / WC_VB);
  const bool states_ready = long_rows >= WC_LONG;
  auto run = [&](auto type, auto ns) {
    using T = decltype(type);
    constexpr int NS = decltype(ns)::value;
    static SharedLimit limits[2];
    const size_t smem = 2 * sizeof(WkvMemory<NS>);
    auto go = [&](auto kernel, SharedLimit& limit) {
      const cudaError_t e = limit.raise(kernel, smem);
      if (e != cudaSuccess) return mlxb_fail((int)e, "wkv_chunks: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
      launch_pdl(kernel, grid, dim3(32 * NS), smem, stream, (const T*)rkv, ld, r_off, k_off, v_off, d_raw, ldd, u, state, slots,
                 token_req, req_first_token, n_requests, o, ldo, H, V, scratch, products, states_ready);
      return mlxb_check_launch("wkv_chunks");
    };
    if (int e = go(wkv_chunks_kernel<T, NS, true>, limits[0])) return e;
    if (long_rows < WC_Q) return 0;                      // no run of two chunks
    if (states_ready) {
      launch_pdl(wkv_states_kernel, dim3(H, n_requests, (V * K + 1023) / 1024), dim3(256), 0, stream, token_req, req_first_token, scratch,
                 (const float*)products, H, V, K);
      if (int e = mlxb_check_launch("wkv_chunks (states)")) return e;
    }
    return go(wkv_chunks_kernel<T, NS, false>, limits[1]);
  };
  auto by_rows = [&](auto type) {
    switch (K) {
      case 16: return run(type, std::integral_constant<int, 1>{});
      case 32: return run(type, std::integral_constant<int, 2>{});
      case 64: return run(type, std::integral_constant<int, 4>{});
      case 128: return run(type, std::integral_constant<int, 8>{});
      default: return run(type, std::integral_constant<int, 16>{});
    }
  };
  if (dtype == MLXB_F32) return by_rows(float{});
  if (dtype == MLXB_BF16) return by_rows(__nv_bfloat16{});
  return mlxb_fail(MLXB_BAD_DTYPE, "wkv_chunks: dtype code %d", dtype);
}

// rkv: [n_tokens, .] (activation dtype) holding r and k (H*K columns each from r_off / k_off) and v (H*V columns from
// v_off); d_raw: float32 [n_tokens, >= H*K] at row stride ldd; u: float32 [H, K]; state: float32 [slots, H, V, K];
// o: float32 [n_tokens, H*V] at row stride ldo.
MLXB_EXPORT int mlxb_wkv_scan(int dtype, const void* rkv, int ld, int r_off, int k_off, int v_off, const float* d_raw,
                              int ldd, const float* u, float* state, const int* slots, const int* token_req,
                              const int* req_first_token, float* o, int ldo, int H, int K, int V, int n_requests,
                              cudaStream_t stream) {
  if (n_requests <= 0) return 0;
  if (H <= 0 || K <= 0 || V <= 0 || K > 32 * WK_NPT || n_requests > 65535)
    return mlxb_fail(MLXB_BAD_ARG, "wkv_scan: %d heads with states of %d x %d (at most %d rows)", H, K, V, 32 * WK_NPT);
  int NS = 1;
  while (NS * WK_NPT < K) NS *= 2;
  // few (request, head) pairs: the columns of a pair over several blocks, never below two warps a block
  const long long pairs = (long long)H * n_requests;
  const int sms = mlxb_sm_count();
  int threads = 2 * pairs >= sms ? 256 : (4 * pairs >= sms ? 128 : 64);
  if (threads < 2 * NS) threads = 2 * NS;
  const int unit = NS >= 32 ? 1 : 32 / NS;                 // columns that make a whole warp
  int VB = threads / NS;
  const int v_up = (V + unit - 1) / unit * unit;
  if (VB > v_up) VB = v_up;
  threads = VB * NS;
  const dim3 grid(H, n_requests, (V + VB - 1) / VB);
  const size_t smem = sizeof(float) * ((size_t)WK_CHUNK * (3 * NS * WK_SEG + VB + 1));
#define WK_GO(T, N)                                                                                                  \
  if (smem > 48 * 1024) {                                                                                            \
    cudaError_t e = cudaFuncSetAttribute(wkv_scan_kernel<T, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e != cudaSuccess) return mlxb_fail((int)e, "wkv_scan: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e)); \
  }                                                                                                                  \
  launch_pdl(wkv_scan_kernel<T, N>, grid, dim3(threads), smem, stream, (const T*)rkv, ld, r_off, k_off, v_off, d_raw, \
             ldd, u, state, slots, token_req, req_first_token, o, ldo, H, K, V, VB)
#define WK_NS(T)                 \
  switch (NS) {                  \
    case 1: WK_GO(T, 1); break;  \
    case 2: WK_GO(T, 2); break;  \
    case 4: WK_GO(T, 4); break;  \
    case 8: WK_GO(T, 8); break;  \
    case 16: WK_GO(T, 16); break; \
    default: WK_GO(T, 32); break; \
  }
  if (dtype == MLXB_F32) { WK_NS(float) }
  else if (dtype == MLXB_BF16) { WK_NS(__nv_bfloat16) }
  else return mlxb_fail(MLXB_BAD_DTYPE, "wkv_scan: dtype code %d", dtype);
#undef WK_NS
#undef WK_GO
  return mlxb_check_launch("wkv_scan");
}
