// Linear layer for many rows (prompt portions) on the 5th-generation tensor cores:
//   C[M,N] = epilogue(A[M,K] . W[N,K]^T + bias[N]) (+ residual[M,N])
// A, W bfloat16 (both operands K-major: the K index is contiguous), C bfloat16 or float32, the residual has C's dtype.
//
// The kernel is persistent: one CTA per SM walks over the 128 x BN output tiles (BN = 32 to 256,
// see tile_choice).  Warp 0 is the TMA producer: it fills a
// ring of shared-memory stages with one or two blocks of 64 of K each, 128x64 tiles of A and BNx64 of W (cp.async.bulk.tensor,
// 128-byte swizzle, completion counted on an mbarrier per stage; rows and columns outside the
// matrices arrive as zeros).  Warp 1 allocates tensor memory and issues tcgen05.mma (kind::f16, bf16
// inputs, float32 accumulator of 128 lanes x BN columns in TMEM), four K=16 steps per block, and
// releases each stage with tcgen05.commit.  There are two accumulators in TMEM: while warps 2-17 (the
// epilogue, four warps per quadrant of 32 TMEM lanes, each a quarter of the columns) read a finished one
// with tcgen05.ld, add the bias, apply gelu_new, add the residual and store, the MMA warp already
// fills the other with the next tile.
// No multicast copy anywhere: every CTA fetches its own tiles.
//
// Pairs (template parameter CG = 2).  The main loop of one CTA is bound by its SM's shared memory: per K step
// 128 rows of A and BN rows of W go in and the tensor core reads the same rows out again, more cycles than the
// products take.  With many rows the kernel therefore runs as thread-block clusters of two CTAs on a
// 256 x BN tile (tcgen05 with .cta_group::2): each CTA fetches its own 128 rows of A and only its half of the
// W rows, the CTA of cluster rank 0 (the leader) issues one product per K step for both, which reads A from
// each CTA's own shared memory and the two halves of W from both, and leaves each CTA's 128 rows of the
// result in that CTA's tensor memory.  The copies of both CTAs are counted on the leader's barrier of the stage
// (.cta_group::2 copies may name a barrier of the peer), a stage is released to both producers by one
// tcgen05.commit that arrives in both CTAs, a finished accumulator is announced to both CTAs' epilogue warps
// the same way, and the epilogue warps of both hand an accumulator back on the leader's barrier.  The tensor
// memory is allocated and freed by warp 1 of both CTAs with the .cta_group::2 forms.  The two CTAs meet at a
// cluster barrier after set-up (so that nobody signals a barrier that is not initialised yet) and before the
// tensor memory is freed (so that nobody frees or leaves while the peer still reads, signals or copies).
//
// Every wait on an mbarrier is bounded: after a limit of polls the waiter raises an abort flag in
// shared memory and a bit in the caller's status word; all roles then fall through to the common
// exit, where the tensor memory is freed.  A timeout therefore ends the kernel with an error code
// instead of a hang.
//
// K and the row strides must be multiples of 8 elements (16 bytes), base addresses 16-byte aligned.
// The accumulation order over K is fixed (block by block, four steps per block), the same in every form, independent of M.
#include <cuda.h>

#include "activations.cuh"
#include "kv_scatter.cuh"
#include "tcgen05.cuh"

MLXB_DEFINE_LAST_ERROR()

constexpr int BM = 128, BK = 64;
constexpr int EPI_WARPS = 16;                     // four per quadrant of TMEM lanes, each a quarter of the columns
constexpr int THREADS = 64 + 32 * EPI_WARPS;
// slices of a tile's columns over the epilogue warps of a quadrant; a tile narrower than 128 leaves warps without work
constexpr int epi_slices(int bn) { return bn >= 128 ? EPI_WARPS / 4 : bn / 32; }
// A stage holds KB blocks of 64 of K, each a tile of its own.
template <int BN, int STAGES, int KB, int CG>
struct Smem {
  alignas(1024) __nv_bfloat16 a[STAGES][KB * BM * BK];
  alignas(1024) __nv_bfloat16 b[STAGES][KB * (BN / CG) * BK];   // in a pair: this CTA's half of the W rows
  alignas(8) uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t drained;       // abort path only: every tensor-core operation issued so far has completed
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) uint4 stage[EPI_WARPS][32 * 4];   // per epilogue warp: 64 bytes of results of each of its 32 rows on their way out
};


// A LayerNorm folded into the weights (see NormFold in gemm_smallm.cuh): the epilogue turns the product of the
// rows as they are into rstd * (sum - mean * colsum[n]).  stats[m] = (mean, rstd) of row m, from row_stats.
struct NormFoldRows {
  const float* colsum;    // [N], null: no fold
  const float2* stats;    // [M]
};

// Results leave through shared memory: a lane holds a row, and written by the lanes that hold them they would be pieces of
// rows 32 rows apart.  A warp puts 64 bytes of each of its 32 rows there (the 16-byte pieces of a row XORed with bits of the row
// number against bank conflicts) and writes them out with four lanes on a row: whole sectors.
__device__ __forceinline__ int stage_index(int row, int piece) { return row * 4 + (piece ^ ((row >> 1) & 3)); }

// 16 bytes of row `row` (an element offset) at column n, from a staged piece.
__device__ __forceinline__ void store_piece(uint4 u, int n, int N, size_t row, float* C) {
  float* out = C + row + n;
  if (n + 4 <= N && ((row + n) & 3) == 0) {
    *reinterpret_cast<uint4*>(out) = u;
  } else {
    const float* e = reinterpret_cast<const float*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n + i < N) out[i] = e[i];
  }
}

// Eight bfloat16 of row `row` (an element offset) at column n8, from a staged piece.
__device__ __forceinline__ void store_piece(uint4 u, int n8, int N, size_t row, __nv_bfloat16* C) {
  __nv_bfloat16* out = C + row + n8;
  if (n8 + 8 <= N && ((row + n8) & 7) == 0) {
    *reinterpret_cast<uint4*>(out) = u;
  } else {
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&u);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (n8 + i < N) out[i] = e[i];
  }
}

// Eight key or value columns n8..n8+7 (n8 >= q_width, a multiple of 8; N = q_width + 2*Hkv*Dh with Dh a
// multiple of 8, so the eight stay inside one head and all of them exist) of one token into the token's page:
// one 16-byte store.  slot: the page's element offset, in_page: the token's row in it.
__device__ __forceinline__ void scatter_piece(uint4 u, int n8, const KvScatter& kv, long long slot, int in_page) {
  const int kvw = kv.Hkv * kv.Dh;
  int c2 = n8 - kv.q_width;
  __nv_bfloat16* pool = kv.k_pool;
  if (c2 >= kvw) { c2 -= kvw; pool = kv.v_pool; }
  const int hh = c2 / kv.Dh, d = c2 - hh * kv.Dh;
  *reinterpret_cast<uint4*>(pool + ((size_t)slot + (size_t)hh * kv.page + in_page) * kv.Dh + d) = u;
}

template <int BN, int STAGES, int KB, typename TO, int EPI, bool SCATTER, int CG>
__global__ void __launch_bounds__(THREADS)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    const float* __restrict__ bias, const __nv_bfloat16* residual, TO* C, int M, int N, int K,
                    int ldc, int* __restrict__ status, KvScatter kv, NormFoldRows fold) {
  extern __shared__ uint8_t smem_raw[];
  Smem<BN, STAGES, KB, CG>& sm = *reinterpret_cast<Smem<BN, STAGES, KB, CG>*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_tiles = (K + KB * BK - 1) / (KB * BK);     // stages a tile; blocks beyond K arrive as zeros
  // A tile is (CG * 128) x BN; in a pair the CTA of rank r takes rows 128 r .. 128 r + 127 of it and fetches rows
  // (BN / 2) r .. of the tile's W rows.  Pair (or CTA) c takes tiles c, c + step, ...
  const int rank = CG == 2 ? (int)cluster_rank() : 0;
  const bool leader = rank == 0;
  const int tiles_m = (M + CG * BM - 1) / (CG * BM), tiles_n = (N + BN - 1) / BN;
  const int n_tiles = tiles_m * tiles_n;
  const int first_tile = (int)blockIdx.x / CG, tile_step = (int)gridDim.x / CG;
  auto tile_m0 = [&](int t) { return (t % tiles_m) * (CG * BM) + rank * BM; };      // this CTA's first row
  auto tile_n0 = [&](int t) { return (t / tiles_m) * BN; };                          // the tile's first column
  constexpr int W_ROWS = BN / CG;                          // W rows per copy
  constexpr uint32_t STAGE_BYTES = CG * KB * (BM + W_ROWS) * BK * sizeof(__nv_bfloat16);   // counted on a stage's barrier
  constexpr uint32_t TMEM_COLS = BN <= 128 ? 2 * BN : 512;   // two accumulators; a power of two

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&sm.acc_full[b], 1); mbar_init(&sm.acc_empty[b], CG * 32 * 4 * epi_slices(BN)); }
    mbar_init(&sm.drained, 1);
    sm.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
  }
  if (warp == 1) {   // the MMA warp owns the tensor memory (in a pair: warp 1 of both CTAs, the same columns in both)
    if (CG == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                   "r"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                   "r"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  volatile int* abort_flag = &sm.abort_flag;
  // In a pair: the leader's barriers as the peer names them, and the peer's abort flag.
  const uint32_t peer_abort = CG == 2 ? peer_addr(&sm.abort_flag, (uint32_t)(rank ^ 1)) : 0u;
  pdl_trigger();
  // The weights do not come from the previous kernel: the W rows of the first tile's first stages are asked
  // for before the wait, so that after it only the rows of A are missing.  The barriers of these stages are armed
  // before the two CTAs of a pair meet, the copies follow after.
  int early = 0;
  if (first_tile < n_tiles) early = k_tiles < STAGES ? k_tiles : STAGES;
  if (threadIdx.x == 0 && leader)
    for (int s = 0; s < early; ++s) mbar_expect_tx(&sm.full[s], STAGE_BYTES);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (CG == 2) cluster_sync();   // the peer's barriers are initialised, the leader's first stages armed
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = sm.tmem_base;
  // this CTA's copies of a stage: its rows of A, its rows of W
  auto load_a = [&](int s, int kt, int m0) {
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
      __nv_bfloat16* dst = sm.a[s] + kb * (BM * BK);
      if (CG == 2) tma_load_2d_pair(dst, &map_a, (kt * KB + kb) * BK, m0, peer_addr(&sm.full[s], 0));
      else tma_load_2d(dst, &map_a, (kt * KB + kb) * BK, m0, &sm.full[s]);
    }
  };
  auto load_w = [&](int s, int kt, int n0) {
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
      __nv_bfloat16* dst = sm.b[s] + kb * (W_ROWS * BK);
      if (CG == 2) tma_load_2d_pair(dst, &map_w, (kt * KB + kb) * BK, n0 + rank * W_ROWS, peer_addr(&sm.full[s], 0));
      else tma_load_2d(dst, &map_w, (kt * KB + kb) * BK, n0, &sm.full[s]);
    }
  };
  if (threadIdx.x == 0)
    for (int s = 0; s < early; ++s) load_w(s, s, tile_n0(first_tile));
  pdl_wait();   // A (and the residual) come from the previous kernel
  residual = after_wait(residual);

  if (warp == 0) {
    int issued = 0;   // stages filled so far, over all tiles
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
      const int m0 = tile_m0(tile), n0 = tile_n0(tile);
      for (int kt = 0; kt < k_tiles; ++kt) {
        if (issued < early) {   // a fresh stage, armed, whose W rows are on their way already
          if (elect_one()) load_a(s, kt, m0);
        } else {
          // free once the products that read it have completed (in a pair: the commit arrives in both CTAs)
          ok = mbar_wait_warp(&sm.empty[s], ph ^ 1, abort_flag, peer_abort);
          if (!ok) break;
          if (elect_one()) {
            if (leader) mbar_expect_tx(&sm.full[s], STAGE_BYTES);
            load_a(s, kt, m0);
            load_w(s, kt, n0);
          }
        }
        ++issued;
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    if (lane == 0 && *abort_flag && leader) {   // gave up: let the copies already issued land before the CTA exits
      for (int i = issued > STAGES ? issued - STAGES : 0; i < issued; ++i) {
        const uint32_t addr = smem_u32(&sm.full[i % STAGES]);
        for (uint32_t p = 0; p < (1u << 20); ++p) {
          uint32_t done;
          asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                       "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(addr), "r"((uint32_t)((i / STAGES) & 1))
                       : "memory");
          if (done) break;
        }
      }
    }
  } else if (warp == 1) {
    if (leader) {   // one thread issues the products, for both CTAs of a pair
      constexpr uint32_t idesc = umma_idesc(CG * BM, BN);
      // the same offsets in both CTAs of a pair: the descriptors name them in each CTA's own shared memory
      const uint64_t da0 = umma_desc(smem_u32(sm.a[0])), db0 = umma_desc(smem_u32(sm.b[0]));
      constexpr uint32_t A_STEP = BM * BK * 2 / 16, B_STEP = W_ROWS * BK * 2 / 16;   // a block, in units of 16 bytes
      int s = 0, it = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++it) {
        const int b = it & 1;
        // the epilogue (of both CTAs) must have drained this accumulator (its previous use was tile it-2)
        ok = mbar_wait_warp(&sm.acc_empty[b], ((it >> 1) & 1) ^ 1, abort_flag, peer_abort);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_acc = tmem_base + (uint32_t)(b * BN);
        for (int kt = 0; kt < k_tiles; ++kt) {
          ok = mbar_wait_warp(&sm.full[s], ph, abort_flag, peer_abort);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = da0 + (uint32_t)(s * KB) * A_STEP, db = db0 + (uint32_t)(s * KB) * B_STEP;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < KB * (BK / 16); ++k) {   // 16 bf16 = 32 bytes = 2 units of the descriptor's start address
              const uint64_t ak = da + (k / (BK / 16)) * A_STEP + 2 * (k % (BK / 16));
              const uint64_t bk = db + (k / (BK / 16)) * B_STEP + 2 * (k % (BK / 16));
              if (CG == 2) umma_bf16_pair(tmem_acc, ak, bk, idesc, (kt > 0 || k > 0) ? 1u : 0u);
              else umma_bf16(tmem_acc, ak, bk, idesc, (kt > 0 || k > 0) ? 1u : 0u);
            }
            // the stage is free once these MMAs have read it
            if (CG == 2) umma_commit_both(&sm.empty[s]);
            else umma_commit(&sm.empty[s]);
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
#ifdef MLXB_TEST_WAIT_TIMEOUT
        if (g_test_withhold_arrival && it == 0) continue;   // the test's missing arrival
#endif
        if (ok && elect_one()) {   // arrives when every MMA of this tile has completed
          if (CG == 2) umma_commit_both(&sm.acc_full[b]);
          else umma_commit(&sm.acc_full[b]);
        }
        __syncwarp();
      }
    }
  } else if (((warp - 2) >> 2) < epi_slices(BN)) {
    // epilogue: warps 2..17; warp w may touch TMEM lanes 32*(w%4) .. +31; the four warps of a quadrant
    // split the tile's columns
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;          // which slice of the columns (0 .. EPI_WARPS/4 - 1)
    constexpr int HALF_COLS = BN / epi_slices(BN);    // 32, 48 or 64 columns per warp
    const uint32_t acc_empty_leader[2] = {CG == 2 ? peer_addr(&sm.acc_empty[0], 0) : 0u,
                                          CG == 2 ? peer_addr(&sm.acc_empty[1], 0) : 0u};
    const TO* res = reinterpret_cast<const TO*>(residual);
    constexpr int PER = 16 / sizeof(TO);               // columns of a 16-byte piece of the output
    uint4* stg = sm.stage[warp - 2];
    const int o_row = lane >> 2, o_piece = lane & 3;   // what this lane writes out: rows o_row + 8 j
    int it = 0;
    for (int tile = first_tile; tile < n_tiles; tile += tile_step, ++it) {
      const int b = it & 1;
      const int m0 = tile_m0(tile) + q * 32, n0 = tile_n0(tile) + half * HALF_COLS;     // this warp's first row and column
      const int m = m0 + lane;
      const bool in = m < M;
      const size_t row = (size_t)m * ldc;
      // While the tile's products run: all that the epilogue needs from memory besides them.  Lane l keeps (bias, column
      // sum) of columns l and l + 32 and hands them around through shared memory chunk by chunk; read from global memory
      // between the steps of the epilogue they cost it a latency each (2048 x 4096 x 1024 with bias, folded norm and
      // gelu_new: 24.3 us, 17.4 without any of them, 19.5 this way).
      float mean = 0.f, rstd = 1.f;
      if (fold.colsum != nullptr && in) {
        const float2 st = fold.stats[m];
        mean = st.x;
        rstd = st.y;
      }
      const float shift = -mean * rstd;
      float2 col_a, col_b;
      {
        const int na = n0 + lane, nb = n0 + 32 + lane;
        const bool oka = na < N && lane < HALF_COLS, okb = nb < N && 32 + lane < HALF_COLS;
        col_a = make_float2(bias != nullptr && oka ? bias[na] : 0.f, fold.colsum != nullptr && oka ? fold.colsum[na] : 0.f);
        col_b = make_float2(bias != nullptr && okb ? bias[nb] : 0.f, fold.colsum != nullptr && okb ? fold.colsum[nb] : 0.f);
      }
      // fused cache write: this row's slot in its page (an element offset before the head and dim are added);
      // -1 for a padding row or an index out of range
      long long slot = -1;
      int in_page = 0;
      if (SCATTER && in && n0 + HALF_COLS > kv.q_width && n0 < N) {
        const int r = kv.token_req[m];
        if (r >= 0) {
          const int pos = kv.positions[m];
          const int lp = pos / kv.page;
          const int pg = (pos >= 0 && lp < kv.max_pages) ? kv.block_table[(size_t)r * kv.max_pages + lp] : -2;
          if (pg == -2) atomicOr(kv.status, MLXB_ST_POSITION_RANGE);
          else if (pg >= kv.n_pages) atomicOr(kv.status, MLXB_ST_PAGE_RANGE);
          else if (pg >= 0) { slot = (long long)pg * kv.Hkv * kv.page; in_page = pos % kv.page; }
        }
      }
      // The residual, four 16-byte pieces a lane.  bfloat16: 32 columns of this lane's row (added before the sum is
      // rounded), a chunk ahead.  float32: the pieces that this lane writes out of 16 columns (added on the way out, four
      // lanes on a row's 64 bytes), half a chunk ahead (2048 x 4096 x 1024: 28.3 us; by rows and in place 40.1).  Bit i of
      // `have`: piece i was fetched (whole and aligned).
      uint4 rp[4];
      unsigned have = 0;
      auto fetch = [&](int c) {       // columns c .. of this warp's
        have = 0;
        if (res == nullptr) return;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int mm = sizeof(TO) == 2 ? m : m0 + o_row + 8 * i;
          const int off = c + (sizeof(TO) == 2 ? i : o_piece) * PER, n = n0 + off;
          const size_t at = (size_t)mm * ldc + n;
          if (mm < M && n + PER <= N && off < HALF_COLS && (at & (PER - 1)) == 0) {
            rp[i] = *reinterpret_cast<const uint4*>(res + at);
            have |= 1u << i;
          }
        }
      };
      fetch(0);
      if (!mbar_wait(&sm.acc_full[b], (it >> 1) & 1, abort_flag, peer_abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + half * HALF_COLS);
#pragma unroll 1
      for (int c0 = 0; c0 < HALF_COLS; c0 += 32) {
        uint32_t r[32];
        if (c0 + 32 <= HALF_COLS) {
          tmem_ld32(taddr + (uint32_t)c0, r);   // every lane takes part
        } else {                                // 48 columns per warp (BN = 192): the last 16
          tmem_ld16(taddr + (uint32_t)c0, r);
        }
        reinterpret_cast<float2*>(stg)[lane] = c0 == 0 ? col_a : col_b;
        __syncwarp();
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 >= HALF_COLS) {   // this warp's part of the accumulator is in registers: hand it back
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          if (CG == 2) mbar_arrive_cluster(acc_empty_leader[b]);   // the leader issues the products into both halves
          else mbar_arrive(&sm.acc_empty[b]);
        }
        float* v = reinterpret_cast<float*>(r);
        const float4* cp = reinterpret_cast<const float4*>(stg);      // (bias, column sum) of two columns: the same for every lane
        if (fold.colsum != nullptr) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float4 c = cp[i];
            v[2 * i] = fmaf(shift, c.y, rstd * v[2 * i]) + c.x;
            v[2 * i + 1] = fmaf(shift, c.w, rstd * v[2 * i + 1]) + c.z;
          }
        } else if (bias != nullptr) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float4 c = cp[i];
            v[2 * i] += c.x;
            v[2 * i + 1] += c.z;
          }
        }
        if (EPI != EPI_NONE) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = activate<EPI, true>(v[i]);
        }
        if (sizeof(TO) == 2 && res != nullptr && in) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if ((have >> i) & 1) {
              const uint32_t w[4] = {rp[i].x, rp[i].y, rp[i].z, rp[i].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                v[8 * i + 2 * e] += __uint_as_float(w[e] << 16);
                v[8 * i + 2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u);
              }
            } else if (c0 + 8 * i < HALF_COLS) {
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (n0 + c0 + 8 * i + e < N) v[8 * i + e] += to_f(res[row + n0 + c0 + 8 * i + e]);
            }
          }
          if (c0 + 32 < HALF_COLS) fetch(c0 + 32);
        }
        __syncwarp();                     // the columns' constants are read before results overwrite them
#pragma unroll
        for (int p0 = 0; p0 < 32; p0 += 4 * PER) {      // 64 bytes of each row at a time
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            uint4 u;
            if (sizeof(TO) == 2) {
              float w[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) w[i] = v[(p * 8 + i) & 31];
              u = pack8(w);
            } else {
              const int i = (p0 + p * 4) & 31;
              u = make_uint4(__float_as_uint(v[i]), __float_as_uint(v[i + 1]), __float_as_uint(v[i + 2]), __float_as_uint(v[i + 3]));
            }
            stg[stage_index(lane, p)] = u;
          }
          __syncwarp();
          const int n = n0 + c0 + p0 + o_piece * PER;
          const bool n_in = c0 + p0 + o_piece * PER < HALF_COLS && n < N;
#pragma unroll
          for (int j = 0; j < 4; ++j) {   // four lanes on a row's 64 bytes, eight rows an instruction
            const int rr = 8 * j + o_row;
            uint4 u = stg[stage_index(rr, o_piece)];
            const int mm = m0 + rr;
            if (sizeof(TO) == 4 && res != nullptr && mm < M && n_in) {
              float* e = reinterpret_cast<float*>(&u);
              if ((have >> j) & 1) {
                e[0] += __uint_as_float(rp[j].x); e[1] += __uint_as_float(rp[j].y);
                e[2] += __uint_as_float(rp[j].z); e[3] += __uint_as_float(rp[j].w);
              } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (n + i < N) e[i] += to_f(res[(size_t)mm * ldc + n + i]);
              }
            }
            long long slot_r = -1;
            int in_page_r = 0;
            if (SCATTER) {   // the row's page, from the lane that looked it up
              slot_r = __shfl_sync(0xffffffffu, slot, rr);
              in_page_r = __shfl_sync(0xffffffffu, in_page, rr);
            }
            if (mm < M && n_in) {
              if (SCATTER && n >= kv.q_width) {
                if (slot_r >= 0) scatter_piece(u, n, kv, slot_r, in_page_r);
              } else {
                store_piece(u, n, N, (size_t)mm * ldc, C);
              }
            }
          }
          if (sizeof(TO) == 4) fetch(c0 + p0 + 16);
          __syncwarp();   // the pieces are read before the next ones overwrite them
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // In a pair nobody goes on alone: the peer's epilogue may still read its tensor memory, and arrivals, copies
  // counted on the leader's barriers and a raised abort flag may still be on their way.
  if (CG == 2) cluster_sync();
  const bool aborted = sm.abort_flag != 0;     // the same in both CTAs of a pair from here on
  if (threadIdx.x == 0 && aborted) atomicOr(status, MLXB_ST_WAIT_TIMEOUT);
  if (warp == 1 && leader) {
    if (aborted && elect_one()) {
      // Somebody gave up.  Products this thread issued may still be running on the tensor memory that is freed
      // below: one more commit arrives when all of them have completed; wait for it, bounded.
      if (CG == 2) umma_commit_pair_local(&sm.drained);
      else umma_commit(&sm.drained);
      const uint32_t addr = smem_u32(&sm.drained);
      for (uint32_t p = 0; p < (1u << 20); ++p) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(addr), "r"(0u) : "memory");
        if (done) break;
      }
    }
    __syncwarp();
  }
  if (CG == 2 && aborted) cluster_sync();   // the peer frees its half only after the leader's products have drained
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (CG == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------- host side

static int make_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(__nv_bfloat16)};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                                            strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    const char* msg = nullptr;
    cuGetErrorString(r, &msg);
    return mlxb_fail(MLXB_BAD_ARG, "linear (tensor cores): cuTensorMapEncodeTiled(%d x %d, ld %d): %s", rows, cols, ld,
                     msg ? msg : "?");
  }
  return 0;
}

static int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  }
  return n;
}

template <int BN, int STAGES, int KB, typename TO, bool SCATTER, int CG>
static int launch(const void* A, const void* W, const float* bias, const void* residual, void* C, int M, int N, int K,
                  int lda, int ldc, int epi, int* status, cudaStream_t stream, const KvScatter& kv, const NormFoldRows& fold) {
  static_assert((BN / CG) % 8 == 0 && BN % (16 * CG) == 0, "a CTA's W rows are whole 8-row swizzle groups");
  static_assert(sizeof(Smem<BN, STAGES, KB, CG>) + 1024 <= 227 * 1024, "stages and staging buffers fit a CTA's shared memory");
  CUtensorMap ma, mw;
  if (int e = make_map(&ma, A, M, K, lda, BM)) return e;
  if (int e = make_map(&mw, W, N, K, K, BN / CG)) return e;      // a copy brings this CTA's rows of the tile
  const size_t smem = sizeof(Smem<BN, STAGES, KB, CG>) + 1024;
  const int n_tiles = ((M + CG * BM - 1) / (CG * BM)) * ((N + BN - 1) / BN);
  const int units = sm_count() / CG;                              // CTAs, or pairs of them
  const dim3 grid(CG * (n_tiles < units ? n_tiles : units));
  // The fused cache write has no activation: only the plain epilogue is built for it.
  return dispatch_activation(SCATTER ? (int)EPI_NONE : epi, [&](auto e) {
    constexpr int EPI = SCATTER ? (int)EPI_NONE : (int)decltype(e)::value;
    auto kern = gemm_tcgen05_kernel<BN, STAGES, KB, TO, EPI, SCATTER, CG>;
    static bool raised = false;   // once per instantiation, and never for the first time inside a stream capture
    if (!raised) {
      cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (err != cudaSuccess) return mlxb_fail((int)err, "linear (tensor cores): %zu bytes of shared memory: %s", smem,
                                               cudaGetErrorString(err));
      raised = true;
    }
    if (CG == 1) {
      launch_pdl(kern, grid, dim3(THREADS), smem, stream, ma, mw, bias, (const __nv_bfloat16*)residual, (TO*)C, M, N, K,
                 ldc, status, kv, fold);
    } else {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = grid;
      cfg.blockDim = dim3(THREADS);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = CG;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      cfg.numAttrs = mlxb_pdl_enabled() ? 2 : 1;
      cudaLaunchKernelEx(&cfg, kern, ma, mw, bias, (const __nv_bfloat16*)residual, (TO*)C, M, N, K, ldc, status, kv, fold);
    }
    return mlxb_check_launch("linear (tensor cores)");
  });
}

// Tile shape and pairs or not: the form whose time, as a sum of what was measured, is least: a launch (set-up, the first copies, the
// last tile's results), every block of 64 of K, every further wave of tiles.  The constants are fits to the times of each form
// at M from 65 to 2048 and N and K from 1024 to 8448, which they give within 5 %.  Single CTAs are best for short K and for up to some
// 2048 of it on wide outputs (2048 x 1024 x 1024: 7.9 us against 8.9; 2048 x 2048 x 2048: 16.1 against 18.2), pairs for many products
// (2048 x 1600 x 6400: 33.9 against 38.0; 2048 x 6400 x 1600: 31.4 against 34.0; 768 x 1600 x 6400: 21.6 against 24.1), and tiles of 64
// or 32 columns where wider ones leave SMs idle (288 x 1280 x 1280: 6.0 against 7.7; 288 x 1280 x 5120: 15.4 against 22.9; 768 x 1024 x
// 1024: 6.0 against 7.1).
// A share of K for each of several CTAs would do more there, but then a row's sums would be added in an order that depends on
// how many rows the call has.
struct TileChoice { int bn, cg; };
struct FormCost { int bn, cg; double launch, block, wave; };      // microseconds
static constexpr FormCost FORMS[] = {{256, 1, 5.35, .288, 2.7}, {192, 1, 5.2, .247, 1.8}, {128, 1, 4.7, .198, 1.4}, {64, 1, 3.9, .174, .6},
                                     {32, 1, 3.4, .160, .5},   {256, 2, 7.1, .288, .9},  {192, 2, 7.35, .216, 1.2}, {128, 2, 6.55, .149, 1.}};
// 128 columns in stages of one block of K: nothing waits less often with two of them where K has no more (2048 x 1024 x 64: 4.3 us
// against 4.8)
static bool short_k(int K) { return K <= 2 * BK; }
static TileChoice tile_choice(int M, int N, int K) {
  // experiments and tests: pairs 0 = never, 1 = wherever there are two row tiles; the width
  const char *want_pair = getenv("MLXB_TC_PAIR"), *want_bn = getenv("MLXB_TC_BN");
  const int sms = sm_count(), steps = (K + BK - 1) / BK;
  TileChoice best = {128, 1};
  double best_cost = -1.;
  for (const FormCost& f : FORMS) {
    if (f.cg == 2 && M <= BM) continue;
    if (want_pair && M > BM && (want_pair[0] == '1') != (f.cg == 2)) continue;
    if (want_bn && atoi(want_bn) != f.bn) continue;
    const long long tiles = (long long)((M + f.cg * BM - 1) / (f.cg * BM)) * ((N + f.bn - 1) / f.bn);
    const int units = sms / f.cg;
    const long long waves = (tiles + units - 1) / units;
    const double launch = f.bn == 128 && f.cg == 1 && short_k(K) ? f.launch - .5 : f.launch;
    const double cost = launch + waves * steps * f.block + (waves - 1) * f.wave;
    if (best_cost < 0. || cost < best_cost) { best = {f.bn, f.cg}; best_cost = cost; }
  }
  return best;
}

// Runs the form that tile_choice took.
template <typename TO, bool SCATTER>
static int launch_choice(const void* A, const void* W, const float* bias, const void* residual, void* C, int M, int N, int K,
                         int lda, int ldc, int epi, int* status, cudaStream_t stream, const KvScatter& kv,
                         const NormFoldRows& fold) {
  const TileChoice t = tile_choice(M, N, K);
#define GO(BN_, ST_, KB_, CG_) \
  return launch<BN_, ST_, KB_, TO, SCATTER, CG_>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, status, stream, kv, fold);
  // stages of two blocks where a block's products take less than what surrounds them (waits, votes and commits, some
  // 0.18 us a stage): 288 x 1280 x 5120 on tiles of 32 columns 15.4 us against 20.1 with stages of one; wider ones gain
  // nothing by it and lose the depth of the ring (pairs of 256 x 192, 2048 x 1600 x 6400: 36.2 against 33.9)
  if (t.cg == 2) {
    if (t.bn == 256) GO(256, 6, 1, 2)
    if (t.bn == 192) GO(192, 6, 1, 2)
    GO(128, 4, 2, 2)
  }
  if (t.bn == 256) GO(256, 4, 1, 1)
  if (t.bn == 192) GO(192, 4, 1, 1)
  if (t.bn == 128 && short_k(K)) GO(128, 4, 1, 1)
  if (t.bn == 128) GO(128, 3, 2, 1)
  if (t.bn == 64) GO(64, 4, 2, 1)
  GO(32, 4, 2, 1)
#undef GO
}

// A: bfloat16 [M, K] at row stride lda; W: bfloat16 [N, K] contiguous; bias float32[N] or null; residual of C's dtype
// [M, N] at row stride ldc or null (may alias C); C bfloat16 or float32 (out_f32) [M, N] at row stride ldc.
// K, lda multiples of 8; A and W 16-byte aligned.  status: int32 word that receives MLXB_ST_WAIT_TIMEOUT if a
// bounded wait inside the kernel gives up.
static int linear_tcgen05(int out_f32, const void* A, const void* W, const float* bias, const void* residual, void* C,
                          int M, int N, int K, int lda, int ldc, int epi, int* status, const NormFoldRows& fold,
                          cudaStream_t stream);

MLXB_EXPORT int mlxb_linear_tcgen05(int out_f32, const void* A, const void* W, const float* bias, const void* residual,
                                    void* C, int M, int N, int K, int lda, int ldc, int epi, int* status,
                                    cudaStream_t stream) {
  return linear_tcgen05(out_f32, A, W, bias, residual, C, M, N, K, lda, ldc, epi, status, NormFoldRows{}, stream);
}

// The same with a folded LayerNorm: W and bias are the folded ones, colsum float32[N], stats float32[M][2]
// (mean, rstd of the rows of A, from mlxb_row_stats).
MLXB_EXPORT int mlxb_linear_tcgen05_fold(int out_f32, const void* A, const void* W, const float* bias,
                                         const void* residual, void* C, int M, int N, int K, int lda, int ldc, int epi,
                                         int* status, const float* colsum, const void* stats, cudaStream_t stream) {
  if (colsum == nullptr || stats == nullptr) return mlxb_fail(MLXB_BAD_ARG, "linear (folded norm): column sums or row statistics missing");
  return linear_tcgen05(out_f32, A, W, bias, residual, C, M, N, K, lda, ldc, epi, status,
                        NormFoldRows{colsum, (const float2*)stats}, stream);
}

static int linear_tcgen05(int out_f32, const void* A, const void* W, const float* bias, const void* residual, void* C,
                          int M, int N, int K, int lda, int ldc, int epi, int* status, const NormFoldRows& fold,
                          cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (K & 7) || (lda & 7) || lda < K || ldc < N)
    return mlxb_fail(MLXB_BAD_ARG, "linear (tensor cores): K %d and row stride %d must be multiples of 8 (ldc %d, N %d)",
                     K, lda, ldc, N);
  if (((uintptr_t)A & 15) || ((uintptr_t)W & 15))
    return mlxb_fail(MLXB_BAD_ARG, "linear (tensor cores): operands must be 16-byte aligned");
  if (!activation_known(epi)) return mlxb_fail(MLXB_BAD_ARG, "linear: epilogue code %d", epi);
  if (out_f32)
    return launch_choice<float, false>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, status, stream, KvScatter{}, fold);
  return launch_choice<__nv_bfloat16, false>(A, W, bias, residual, C, M, N, K, lda, ldc, epi, status, stream, KvScatter{}, fold);
}


// The fused [q | k | v] projection with the cache write in its epilogue, for many rows: columns [0, q_width) go
// to C (bfloat16, row stride ldc); key and value columns go into k_pool / v_pool [n_pages, Hkv, page, Dh] at each
// token's page and row.  N = q_width + 2*Hkv*Dh; q_width and Dh multiples of 8.  Rows with token_req < 0 write
// no keys or values.
static int linear_tcgen05_qkv(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, int lda,
                              int ldc, const int* positions, const int* token_req, const int* block_table,
                              int max_pages, int n_pages, int page, int Hkv, int Dh, int q_width, void* k_pool,
                              void* v_pool, int* status, const NormFoldRows& fold, cudaStream_t stream);

MLXB_EXPORT int mlxb_linear_tcgen05_qkv(const void* A, const void* W, const float* bias, void* C, int M, int N, int K,
                                        int lda, int ldc, const int* positions, const int* token_req,
                                        const int* block_table, int max_pages, int n_pages, int page, int Hkv, int Dh,
                                        int q_width, void* k_pool, void* v_pool, int* status, cudaStream_t stream) {
  return linear_tcgen05_qkv(A, W, bias, C, M, N, K, lda, ldc, positions, token_req, block_table, max_pages, n_pages,
                            page, Hkv, Dh, q_width, k_pool, v_pool, status, NormFoldRows{}, stream);
}

// The same with a folded LayerNorm (see mlxb_linear_tcgen05_fold).
MLXB_EXPORT int mlxb_linear_tcgen05_qkv_fold(const void* A, const void* W, const float* bias, void* C, int M, int N,
                                             int K, int lda, int ldc, const int* positions, const int* token_req,
                                             const int* block_table, int max_pages, int n_pages, int page, int Hkv,
                                             int Dh, int q_width, void* k_pool, void* v_pool, int* status,
                                             const float* colsum, const void* stats, cudaStream_t stream) {
  if (colsum == nullptr || stats == nullptr) return mlxb_fail(MLXB_BAD_ARG, "linear (folded norm): column sums or row statistics missing");
  return linear_tcgen05_qkv(A, W, bias, C, M, N, K, lda, ldc, positions, token_req, block_table, max_pages, n_pages,
                            page, Hkv, Dh, q_width, k_pool, v_pool, status, NormFoldRows{colsum, (const float2*)stats},
                            stream);
}

static int linear_tcgen05_qkv(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, int lda,
                              int ldc, const int* positions, const int* token_req, const int* block_table,
                              int max_pages, int n_pages, int page, int Hkv, int Dh, int q_width, void* k_pool,
                              void* v_pool, int* status, const NormFoldRows& fold, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (K & 7) || (lda & 7) || lda < K || ldc < N)
    return mlxb_fail(MLXB_BAD_ARG, "linear (tensor cores): K %d and row stride %d must be multiples of 8 (ldc %d, N %d)",
                     K, lda, ldc, N);
  if (((uintptr_t)A & 15) || ((uintptr_t)W & 15) || ((uintptr_t)k_pool & 15) || ((uintptr_t)v_pool & 15))
    return mlxb_fail(MLXB_BAD_ARG, "linear (tensor cores): operands must be 16-byte aligned");
  if (Hkv <= 0 || Dh <= 0 || (Dh & 7) || page <= 0 || q_width < 0 || (q_width & 7) || N != q_width + 2 * Hkv * Dh)
    return mlxb_fail(MLXB_BAD_ARG, "linear (q|k|v): %d outputs for %d query columns and 2 x %d x %d", N, q_width, Hkv, Dh);
  const KvScatter kv = {positions, token_req, block_table, (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, status,
                        max_pages, n_pages, page, Hkv, Dh, q_width};
  return launch_choice<__nv_bfloat16, true>(A, W, bias, nullptr, C, M, N, K, lda, ldc, EPI_NONE, status, stream, kv, fold);
}
