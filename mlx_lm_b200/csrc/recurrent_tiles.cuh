// What the recurrences that run in tiles of rows on tensor cores share: how long a request's run of rows is, and staging of
// one head's rows in shared memory.
#pragma once

#include "common.cuh"

// Rows t0 .. t1-1 that belong to request r (they come first in the range).  Every thread of the block calls it.
__device__ __forceinline__ int run_length(const int* __restrict__ token_req, int t0, int t1, int r) {
  int n = 0;
  for (int base = t0; base < t1; base += 4 * blockDim.x) {      // four loads on their way together
    bool mine[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = base + i * blockDim.x + threadIdx.x;
      mine[i] = t < t1 && token_req[t] == r;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (base + i * (int)blockDim.x < t1) n += __syncthreads_count(mine[i]);
  }
  return n;
}

// A request's run of rows goes through a recurrence token by token or in chunks of 64 rows, whichever takes less time by this
// rule (nanoseconds of a launch, from the layer's sizes and the number of requests with runs; what is known of the times
// stands with the rule's maker, ops.chunk_rule).  A single row never goes in chunks.
struct ChunkRule {
  int scan_fixed, scan_row, chunk_fixed, chunk_each;
  __device__ __forceinline__ bool chunks(int n) const {
    return n > 1 && chunk_fixed + (long long)chunk_each * ((n + 63) / 64) < scan_fixed + (long long)scan_row * n;
  }
};

// Job `job` of the step: chunk c (of `rows` rows) of request r, in the order of the requests (all, or those listed; -1: none); base: chunks before the request's last ones, of the
// requests before it (where its states between chunks are kept).  r = -1: there are fewer jobs.  A whole warp calls it.
__device__ __forceinline__ int listed_request(const int* __restrict__ requests, int n_requests, int i) {
  return i >= n_requests ? -1 : requests != nullptr ? requests[i] : i;
}
struct ChunkJob { int r, c, base; };
__device__ __forceinline__ ChunkJob find_job(const int* __restrict__ req_first_token, const int* __restrict__ requests, int n_requests,
                                             int job, int rows) {
  const int lane = threadIdx.x & 31;
  ChunkJob out = {-1, 0, 0};
  int before = 0;
  for (int r0 = 0; r0 < n_requests; r0 += 32) {
    const int r = listed_request(requests, n_requests, r0 + lane);
    const int mine = r >= 0 ? (req_first_token[r + 1] - req_first_token[r] + rows - 1) / rows : 0;
    int jobs = mine, kept = mine > 0 ? mine - 1 : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, jobs, o), w = __shfl_up_sync(0xffffffffu, kept, o);
      if (lane >= o) { jobs += u; kept += w; }
    }
    const unsigned hit = __ballot_sync(0xffffffffu, before + jobs > job);
    if (hit) {
      const int src = __ffs(hit) - 1;
      out.r = __shfl_sync(0xffffffffu, r, src);
      out.c = job - before - __shfl_sync(0xffffffffu, jobs - mine, src);
      out.base += __shfl_sync(0xffffffffu, kept - (mine > 0 ? mine - 1 : 0), src);
      return out;
    }
    before += __shfl_sync(0xffffffffu, jobs, 31);
    out.base += __shfl_sync(0xffffffffu, kept, 31);
  }
  return out;
}
// The jobs of the listed requests before number i.  A whole warp calls it.
__device__ __forceinline__ int jobs_before(const int* __restrict__ req_first_token, const int* __restrict__ requests, int i, int rows) {
  int jobs = 0;
  for (int r0 = 0; r0 < i; r0 += 32) {
    const int r = listed_request(requests, i, r0 + (threadIdx.x & 31));
    jobs += r >= 0 ? (req_first_token[r + 1] - req_first_token[r] + rows - 1) / rows : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) jobs += __shfl_xor_sync(0xffffffffu, jobs, o);
  return jobs;
}

// Rows of v: columns v0 .. v0 + VS - 1 of one head into [rows, lds]; zeros beyond n rows and beyond V columns.
template <bool VEC>
__device__ __forceinline__ void stage_values(const __nv_bfloat16* src, int ld, int row0, int n, int rows, int v0, int V, int VS,
                                             __nv_bfloat16* sv, int lds) {
  if (VEC) {
    const int per = VS / 8;
#pragma unroll 4
    for (int e = threadIdx.x; e < rows * per; e += blockDim.x) {
      const int tok = e / per, c = (e - tok * per) * 8;
      uint4 u = make_uint4(0u, 0u, 0u, 0u);
      if (tok < n && v0 + c < V) u = *reinterpret_cast<const uint4*>(src + (size_t)(row0 + tok) * ld + v0 + c);
      *reinterpret_cast<uint4*>(sv + tok * lds + c) = u;
    }
  } else {
    for (int e = threadIdx.x; e < rows * VS; e += blockDim.x) {
      const int tok = e / VS, c = e - tok * VS;
      sv[tok * lds + c] = (tok < n && v0 + c < V) ? src[(size_t)(row0 + tok) * ld + v0 + c] : __float2bfloat16_rn(0.f);
    }
  }
}
