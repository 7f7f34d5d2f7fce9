// The attention of attention_wide.cu for prompt portions on the 5th-generation tensor cores (bfloat16 pages, float32
// accumulation): scores mixed across heads, latent rows whose first columns are the values, wide heads, masks by window, by runs of
// positions and with kept first positions, soft caps and gates, with attention_wide_tc.cu's arithmetic: queries in float32 as two
// bfloat16 halves (hi + lo), mixed queries against a token's key heads side by side, blocks of 64 keys that start at multiples of
// 64 (kept first positions first), weights rounded to bfloat16 and summed as rounded.
//
// A CTA has 128 rows: TQ = 128 / HG consecutive tokens of one request times HG neighbouring heads that share a value head.
// What bounds it is a tile's chain of blocks: S = Q K^T is DkE / 16 steps of two products 128 x 64 x 16 (hi and lo), O += P V
// another 4 Dv / 64, and the softmax of 128 x 64 scores; so a block's products run during the softmax of the block before, and
// keys arrive two blocks ahead.  With mma.sync (attention_wide_tc.cu) a CTA of 64 rows reads a fragment of shared memory for every
// product.  2027 rows in portions of 731, 683 and 613, mma.sync and here, inputs in L2: mixed scores of 16 heads 245 and 82 us, of 32
// heads 1342 and 217, latent rows 200 and 83 (16 heads), 394 and 168 (32).  A tile takes 20 us and 3 to 4 a block of keys.
//
//   warp 9       producer: the pages of a block, a TMA copy per page and chunk of 64 columns, into a ring of 8 KB slots
//                ([64 keys][64 columns], 128-byte swizzle)
//   warp 8       issues the products.  A of the low halves lies in tensor memory (32 columns a chunk of 64, as far as they go, the
//                rest beside the high halves in shared memory), P in tensor memory in place of its scores, V as it lies in the
//                pages (MN-major; the key chunks themselves where the values are their first columns)
//   warps 0-7    mix and take apart the queries, then the softmax, two threads a row (32 of a block's 64 keys each).  O stays in
//                tensor memory: it is scaled only when a row's maximum has grown by more than 2^8 since the last time, which no
//                result depends on (weights and their sum refer to the same maximum), each row by itself
//
// Keys of a block that no query of the tile sees (behind the window, beyond the last position) are there as zeros among the values:
// the softmax warps clear them, so that what earlier owners left in a page reaches nobody.  Keys that some query of the tile sees must
// have finite values: to the others they are zero times the value, so an infinity or a NaN spoils the up to 128 / HG - 1 tokens
// of the same request before it in its tile (as with mma.sync, whose tiles have 64 rows).  The order of additions for a row depends on
// its position only.  Weights are 2^x by ex2.approx (two units in the last place) before they are rounded to bfloat16.
//
// Every wait on an mbarrier is bounded (tcgen05.cuh); after the limit all roles leave their loops, the copies and products in
// flight are waited for, bounded, and MLXB_ST_WAIT_TIMEOUT is reported.
#include "tcgen05.cuh"

MLXB_DEFINE_LAST_ERROR()

constexpr int M = 128, KB = 64;                     // rows of a CTA, keys of a block
constexpr int SOFT_WARPS = 8, SOFT_THREADS = 32 * SOFT_WARPS;
constexpr int MMA_WARP = SOFT_WARPS, LOAD_WARP = SOFT_WARPS + 1;
constexpr int THREADS = SOFT_THREADS + 64;
constexpr int MAX_SLOTS = 20;
constexpr int Q_CHUNK = M * 64 * 2, SLOT = KB * 64 * 2;      // bytes of 64 columns of the queries, of a block's keys or values
constexpr int MAX_MIX = 512;                        // numbers of the mixing matrix that a CTA keeps
constexpr int STALE = 8;                            // powers of two that a row's maximum may grow before O is scaled

struct Control {
  uint64_t full[MAX_SLOTS], empty[MAX_SLOTS];
  uint64_t s_full[2], p_full[2], o_full;           // by block & 1: a pair of softmax warps may be a block ahead of another
  uint64_t x_full[4];                               // exchange between the two warps of the same rows
  uint64_t drained;                                 // abort path only
  float row_max[2][2][M];                           // [block & 1][half][row]
  float talk[MAX_MIX];                              // the mixing matrix's rows of the CTA's heads
  uint32_t tmem_base;
  int abort_flag;
};

struct WideArgs {
  const float* q;
  const int* tiles;
  const int* block_table;
  const float* talk;
  const __nv_bfloat16* gate;
  void* out;
  int* status;
  int ldq, qhs, subs, n_tiles, max_pages, n_pages, page, Hq, Hkv, Hv, Dk, Dv, window, chunk, ldg, ldo, ohs, keep_first, gate_cols;
  int HG, steps, chunks, v_chunks, lo_tmem, slots, shared_v, tmem_cols, vec_out, mix_fast;
  float scale, softcap;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// A (the low halves, or P) in tensor memory
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
// Loads with their wait in one statement: between two statements the compiler may put arithmetic on registers that the load
// has not written yet.
#define LD_REGS_16 "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15"
__device__ __forceinline__ void tmem_get16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {" LD_REGS_16 "}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_get32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {" LD_REGS_16
               ", %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
               "tcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
                 "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
                 "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ int stage_index(int row, int piece) { return row * 4 + (piece ^ ((row >> 1) & 3)); }

// A mark on the ring: the slot a block starts at, and how often the ring has gone round before it (mod 2).
struct Mark {
  int slot;
  uint32_t ph;
  __device__ __forceinline__ void step(int n, int slots) {
    slot += n;
    if (slot >= slots) { slot -= slots; ph ^= 1u; }
  }
};

template <typename TO>
__global__ void __launch_bounds__(THREADS, 1)
attention_wide_tcgen05_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                              const __grid_constant__ WideArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* s_hi = base;                                            // [chunk][128 rows][64], swizzled
  uint8_t* s_lo = s_hi + a.chunks * Q_CHUNK;                       // the low halves that tensor memory has no room for
  uint8_t* ring = s_lo + (a.chunks - a.lo_tmem) * Q_CHUNK;
  Control& sm = *reinterpret_cast<Control*>(ring + a.slots * SLOT);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int HG = a.HG, TQ = M / HG, hg_shift = __ffs(HG) - 1;
  // tiles come longest chain first; within one the last tokens have the longest
  const int tile = blockIdx.x / a.subs, sub = a.subs - 1 - ((int)blockIdx.x - tile * a.subs);
  const int t_first = a.tiles[4 * tile], n_tile = a.tiles[4 * tile + 1], bt_row = a.tiles[4 * tile + 2];
  const int nq = min(TQ, n_tile - sub * TQ);
  if (nq <= 0) return;
  const int t0 = t_first + sub * TQ, pos0 = a.tiles[4 * tile + 3] + sub * TQ;
  const int h0 = blockIdx.y * HG, rep = a.Hq / a.Hkv, ck = h0 / rep, cv = ck / (a.Hkv / a.Hv);
  const int* bt = a.block_table + (size_t)bt_row * a.max_pages;
  int lo_min = 0;                                                  // the first key that the tile's first token sees
  if (a.window > 0 && pos0 - a.window + 1 > lo_min) lo_min = pos0 - a.window + 1;
  if (a.chunk > 0 && (pos0 / a.chunk) * a.chunk > lo_min) lo_min = (pos0 / a.chunk) * a.chunk;
  const int last_pos = pos0 + nq - 1;
  const int kb_lo = lo_min / KB, kb_hi = last_pos / KB;
  const int kept = min(a.keep_first, lo_min), kept_blocks = min((kept + KB - 1) / KB, kb_lo);
  const int n_blocks = kept_blocks + kb_hi - kb_lo + 1;
  auto kb_at = [&](int i) { return i < kept_blocks ? i : kb_lo + i - kept_blocks; };
  const int per_block = a.chunks + (a.shared_v ? 0 : a.v_chunks);

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.slots; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&sm.s_full[b], 1); mbar_init(&sm.p_full[b], SOFT_WARPS); }
    mbar_init(&sm.o_full, 1);
    for (int w = 0; w < 4; ++w) mbar_init(&sm.x_full[w], 2);
    mbar_init(&sm.drained, 1);
    sm.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
  }
  if (a.mix_fast)
    for (int e = threadIdx.x; e < HG * a.Hq; e += THREADS) sm.talk[e] = a.talk[h0 * a.Hq + e];
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(a.tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // tensor memory: two buffers of 64 columns (scores, then P in the first 32), the low halves, O
  const uint32_t tmem_s = sm.tmem_base, tmem_lo = tmem_s + 2 * KB, tmem_o = tmem_lo + 32u * a.lo_tmem;
  volatile int* abort_flag = &sm.abort_flag;
  pdl_trigger();
  pdl_wait();

  // ---- the queries: mixed in float32, taken apart; low halves on their way to tensor memory pass through the ring
  {
    const float* q = after_wait(a.q);
    const int room = a.slots / 2;                                  // chunks of queries that fit the ring
    // Rows of no token are zeros, but with a cap the last token's: capping a score of zero is a quotient of zero, 370 cycles, and a tile
    // with such rows took twice its time (130 tokens at 1900 positions, 8 heads of 64: 272 us, 133 this way).
    const int n_rows = a.softcap > 0.f ? TQ : nq;
    for (int c0 = 0; c0 < a.chunks; c0 += room) {
      const int n_c = min(room, a.chunks - c0), per_row = n_c * 16;
      if (c0 > 0) __syncthreads();
      if (threadIdx.x < SOFT_THREADS) {
        auto put = [&](int r, int col, const float4& v) {      // four columns of a row, as halves
          const float f[4] = {v.x, v.y, v.z, v.w};
          __nv_bfloat162 hi[2], lo[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            hi[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
            const float2 b = __bfloat1622float2(hi[i]);
            lo[i] = __floats2bfloat162_rn(f[2 * i] - b.x, f[2 * i + 1] - b.y);
          }
          const int j = col >> 6, cc = col & 63;
          const uint32_t at = (uint32_t)r * 128 + ((uint32_t)((cc >> 3) ^ (r & 7)) << 4) + (cc & 4) * 2;
          *reinterpret_cast<uint2*>(s_hi + j * Q_CHUNK + at) = *reinterpret_cast<const uint2*>(hi);
          uint8_t* dst = j < a.lo_tmem ? ring + (j - c0) * Q_CHUNK : s_lo + (j - a.lo_tmem) * Q_CHUNK;
          *reinterpret_cast<uint2*>(dst + at) = *reinterpret_cast<const uint2*>(lo);
        };
        // Every thread asks for eight pieces before it uses the first: one after the other (a store of the one in front of the
        // load of the next) they were half of the kernel's time.
        if (a.mix_fast) {      // a piece of all heads of a key head gives a piece of each of the CTA's rows of its token
          const int items = TQ * 16 * n_c;
          for (int e0 = threadIdx.x; e0 < items; e0 += 2 * SOFT_THREADS) {
            float4 u[2][4];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const int e = e0 + k * SOFT_THREADS, x = e / (TQ * 16), y = e - x * (TQ * 16), tq = y >> 4, col = (c0 + x) * 64 + (y & 15) * 4;
              const int c = col / a.Dk, d = col - c * a.Dk;
              const bool in = e < items && tq < n_rows && c < a.Hkv;
              const float* qt = q + (size_t)(t0 + min(tq, nq - 1)) * a.ldq + (size_t)(c * rep) * a.qhs + d;
#pragma unroll
              for (int i = 0; i < 4; ++i)
                u[k][i] = in && i < rep ? *reinterpret_cast<const float4*>(qt + (size_t)i * a.qhs) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const int e = e0 + k * SOFT_THREADS, x = e / (TQ * 16), y = e - x * (TQ * 16), tq = y >> 4, col = (c0 + x) * 64 + (y & 15) * 4;
              const int c = min(col / a.Dk, a.Hkv - 1);
              if (e >= items) continue;
              for (int hh = 0; hh < HG; ++hh) {
                const float* w = sm.talk + hh * a.Hq + c * rep;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const float f = i < rep ? w[i] : 0.f;
                  if (i < rep) {
                    v.x = fmaf(f, u[k][i].x, v.x); v.y = fmaf(f, u[k][i].y, v.y);
                    v.z = fmaf(f, u[k][i].z, v.z); v.w = fmaf(f, u[k][i].w, v.w);
                  }
                }
                put(tq * HG + hh, col, v);
              }
            }
          }
        } else if (a.talk == nullptr) {
          const int items = M * per_row;
          for (int e0 = threadIdx.x; e0 < items; e0 += 8 * SOFT_THREADS) {
            float4 u[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int e = e0 + k * SOFT_THREADS, r = e / per_row, col = c0 * 64 + (e - r * per_row) * 4, tq = r >> hg_shift;
              u[k] = e < items && tq < n_rows && col < a.Dk
                         ? *reinterpret_cast<const float4*>(q + (size_t)(t0 + min(tq, nq - 1)) * a.ldq + (size_t)(h0 + (r & (HG - 1))) * a.qhs + col)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int e = e0 + k * SOFT_THREADS, r = e / per_row;
              if (e < items) put(r, c0 * 64 + (e - r * per_row) * 4, u[k]);
            }
          }
        } else {
          for (int e = threadIdx.x; e < M * per_row; e += SOFT_THREADS) {
            const int r = e / per_row, col = c0 * 64 + (e - r * per_row) * 4;
            const int tq = r >> hg_shift, h = h0 + (r & (HG - 1)), c = col / a.Dk, d = col - c * a.Dk;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tq < n_rows && c < a.Hkv) {
              const float* qt = q + (size_t)(t0 + min(tq, nq - 1)) * a.ldq;
              for (int i = 0; i < rep; ++i) {
                const float w = __ldg(a.talk + h * a.Hq + c * rep + i);
                const float4 u = *reinterpret_cast<const float4*>(qt + (size_t)(c * rep + i) * a.qhs + d);
                v.x = fmaf(w, u.x, v.x); v.y = fmaf(w, u.y, v.y); v.z = fmaf(w, u.z, v.z); v.w = fmaf(w, u.w, v.w);
              }
            }
            put(r, col, v);
          }
        }
      }
      __syncthreads();
      if (warp < SOFT_WARPS) {      // a thread's half row of a chunk: 32 columns, 16 of tensor memory
        const int half = warp >> 2, r = (warp & 3) * 32 + lane;
        for (int j = c0; j < min(c0 + n_c, a.lo_tmem); ++j) {
          uint32_t w[16];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const uint4 u = *reinterpret_cast<const uint4*>(ring + (j - c0) * Q_CHUNK + r * 128 + (((half * 4 + p) ^ (r & 7)) << 4));
            w[4 * p] = u.x; w[4 * p + 1] = u.y; w[4 * p + 2] = u.z; w[4 * p + 3] = u.w;
          }
          tmem_st16(tmem_lo + ((uint32_t)((warp & 3) * 32) << 16) + 32u * j + 16u * half, w);
        }
        tmem_wait_st();
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the products and the copies see (and follow) ordinary accesses
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }

  if (warp == LOAD_WARP) {
    const int page = a.page, shift = __ffs(page) - 1, ppb = KB / page;
    // Pages that a block covers but no query of the tile can see (the cache may have given them back) are loaded from the page
    // of the tile's first query instead.
    int first_page = (pos0 >> shift) < a.max_pages ? bt[pos0 >> shift] : -1;
    if (first_page < 0 || first_page >= a.n_pages) {
      if (lane == 0) atomicOr(a.status, first_page < 0 ? MLXB_ST_POSITION_RANGE : MLXB_ST_PAGE_RANGE);
      first_page = 0;
    }
    auto page_of = [&](int i) {
      int pg = first_page;
      const int key0 = i < n_blocks ? kb_at(i) * KB + lane * page : last_pos + 1;
      if (lane < ppb && key0 <= last_pos && (key0 + page > lo_min || key0 < kept)) {
        const int lp = key0 >> shift;
        const int id = lp < a.max_pages ? bt[lp] : -1;
        if (id < 0 || id >= a.n_pages) atomicOr(a.status, id < 0 ? MLXB_ST_POSITION_RANGE : MLXB_ST_PAGE_RANGE);
        else pg = id;
      }
      return pg;
    };
    Mark at = {0, 0u};
    int issued = 0;
    bool ok = true;
    int pg = page_of(0);
    for (int i = 0; i < n_blocks && ok; ++i) {
      const int pg_next = page_of(i + 1);
      for (int c = 0; c < per_block; ++c) {
        ok = mbar_wait_warp(&sm.empty[at.slot], at.ph ^ 1u, abort_flag);
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(&sm.full[at.slot], SLOT);
        __syncwarp();
        if (lane < ppb) {
          uint8_t* dst = ring + at.slot * SLOT + lane * page * 128;
          if (c < a.chunks) {
            const int head = a.talk != nullptr ? 64 * c / a.Dk : ck, col = a.talk != nullptr ? 64 * c % a.Dk : 64 * c;
            tma_load_2d(dst, &map_k, col, (pg * a.Hkv + head) * page, &sm.full[at.slot]);
          } else {
            tma_load_2d(dst, &map_v, 64 * (c - a.chunks), (pg * a.Hv + cv) * page, &sm.full[at.slot]);
          }
        }
        ++issued;
        at.step(1, a.slots);
      }
      pg = pg_next;
    }
    if (*abort_flag && lane == 0) {      // gave up: the copies already issued land before the CTA ends
      for (int i = max(0, issued - a.slots); i < issued; ++i) {
        const uint32_t addr = smem_u32(&sm.full[i % a.slots]);
        for (uint32_t p = 0; p < (1u << 20); ++p) {
          uint32_t done;
          asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                       "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(addr), "r"((uint32_t)((i / a.slots) & 1)) : "memory");
          if (done) break;
        }
      }
    }
  } else if (warp == MMA_WARP) {
    constexpr uint32_t idesc_s = umma_idesc(M, KB), idesc_o = umma_idesc(M, 64) | (1u << 16);      // B of O: MN-major
    const uint64_t d_hi = umma_desc(smem_u32(s_hi)), d_lo = umma_desc(smem_u32(s_lo)), d_ring = umma_desc(smem_u32(ring));
    Mark s_at = {0, 0u}, v_at = {0, 0u};                           // where the next block of S, and of V, starts
    if (!a.shared_v) v_at.step(a.chunks, a.slots);
    bool ok = true;
    auto issue_s = [&](int i) {
      Mark at = s_at;
      for (int c = 0; c < a.chunks; ++c) {
        ok = mbar_wait_warp(&sm.full[at.slot], at.ph, abort_flag);
        if (!ok) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint32_t d = tmem_s + (uint32_t)((i & 1) * KB);
          const uint64_t dk = d_ring + (uint32_t)(at.slot * (SLOT / 16));
          const int n = min(4, a.steps - 4 * c);
          for (int k = 0; k < n; ++k) {
            if (c < a.lo_tmem) umma_bf16_ta(d, tmem_lo + 32u * c + 8u * k, dk + 2 * k, idesc_s, c + k > 0 ? 1u : 0u);
            else umma_bf16(d, d_lo + (uint32_t)((c - a.lo_tmem) * (Q_CHUNK / 16) + 2 * k), dk + 2 * k, idesc_s, c + k > 0 ? 1u : 0u);
          }
          for (int k = 0; k < n; ++k) umma_bf16(d, d_hi + (uint32_t)(c * (Q_CHUNK / 16) + 2 * k), dk + 2 * k, idesc_s, 1u);
          if (!a.shared_v || c >= a.v_chunks) umma_commit(&sm.empty[at.slot]);
#ifdef MLXB_TEST_WAIT_TIMEOUT
          if (!g_test_withhold_arrival || i > 0)       // the test's missing arrival
#endif
          if (c + 1 == a.chunks) umma_commit(&sm.s_full[i & 1]);
        }
        __syncwarp();
        at.step(1, a.slots);
      }
      s_at.step(per_block, a.slots);
    };
    issue_s(0);
    for (int i = 0; i < n_blocks && ok; ++i) {
      if (i + 1 < n_blocks) {      // its buffer held P(i - 1)
        if (i > 0 && !(ok = mbar_wait_warp(&sm.o_full, (uint32_t)((i - 1) & 1), abort_flag))) break;
        issue_s(i + 1);
        if (!ok) break;
      }
      if (!(ok = mbar_wait_warp(&sm.p_full[i & 1], (uint32_t)((i >> 1) & 1), abort_flag))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      Mark at = v_at;
      for (int c = 0; c < a.v_chunks; ++c) {
        if (!(ok = mbar_wait_warp(&sm.full[at.slot], at.ph, abort_flag))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < KB / 16; ++j)      // 16 keys a step: 8 columns of P, 16 rows of V
            umma_bf16_ta(tmem_o + 64u * c, tmem_s + (uint32_t)((i & 1) * KB) + 8u * j,
                         d_ring + (uint32_t)(at.slot * (SLOT / 16) + j * (16 * 128 / 16)), idesc_o, i + j > 0 ? 1u : 0u);
          umma_commit(&sm.empty[at.slot]);
          if (c + 1 == a.v_chunks) umma_commit(&sm.o_full);
        }
        __syncwarp();
        at.step(1, a.slots);
      }
      v_at.step(per_block, a.slots);
    }
  } else {
    const int half = warp >> 2, r = (warp & 3) * 32 + lane;
    const int tq = r >> hg_shift, pos = tq < nq ? pos0 + tq : -1;
    int lo = 0;                                                    // the row's own first key
    if (a.window > 0 && pos - a.window + 1 > lo) lo = pos - a.window + 1;
    if (a.chunk > 0 && (pos / a.chunk) * a.chunk > lo) lo = (pos / a.chunk) * a.chunk;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const int o_cols = a.v_chunks * 32, o_first = half * o_cols;  // this thread's columns of O
    const float mult = a.softcap > 0.f ? 1.4426950408889634f : a.scale * 1.4426950408889634f;
    uint64_t* x_full = &sm.x_full[warp & 3];
    float m = -INFINITY, l = 0.f;      // what the weights refer to (units of log2), the sum of this half's weights
    Mark v_at = {0, 0u};
    if (!a.shared_v) v_at.step(a.chunks, a.slots);
    bool ok = true;
    int i = 0;
    for (; i < n_blocks; ++i) {
      const int j0 = kb_at(i) * KB, jh = j0 + 32 * half;
      const uint32_t t_s = tmem_s + lanes + (uint32_t)((i & 1) * KB);
      if (!(ok = mbar_wait_warp(&sm.s_full[i & 1], (uint32_t)((i >> 1) & 1), abort_flag))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t s[32];
      tmem_get32(t_s + 32u * half, s);
      const bool open = j0 + KB - 1 <= pos0 && (j0 >= lo_min || j0 + KB <= kept);      // every key is visible to the first token
      // (and to the others, unless the window or the run moves on between them)
      const bool all = open && (a.window <= 0 || j0 >= last_pos - a.window + 1 || j0 + KB <= kept) &&
                       (a.chunk <= 0 || j0 >= last_pos / a.chunk * a.chunk);
      float v[32], mx = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        float f = __uint_as_float(s[e]);
        if (a.softcap > 0.f) f = a.softcap * tanhf(f * a.scale / a.softcap);
        v[e] = f * mult;
      }
      __syncwarp();
      if (!all) {
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const int j = jh + e;
          if (!(j <= pos && (j >= lo || j < a.keep_first))) v[e] = -INFINITY;
        }
      }
#pragma unroll
      for (int e = 0; e < 32; e += 2) { mx = fmaxf(mx, v[e]); mx1 = fmaxf(mx1, v[e + 1]); }
      sm.row_max[i & 1][half][r] = fmaxf(mx, mx1);
      __syncwarp();
      if (lane == 0) mbar_arrive(x_full);
      if (!(ok = mbar_wait_warp(x_full, (uint32_t)(i & 1), abort_flag))) break;
      const float top = fmaxf(m, fmaxf(sm.row_max[i & 1][0][r], sm.row_max[i & 1][1][r]));
      // O and the sum refer to m until it is out of date
      const bool grown = top > m + (float)STALE && m != -INFINITY;
      const float corr = grown ? fast_exp2(m - top) : 1.f;
      if (grown || m == -INFINITY) m = top;
      if (i > 0 && __any_sync(0xffffffffu, grown)) {
        if (!(ok = mbar_wait_warp(&sm.o_full, (uint32_t)((i - 1) & 1), abort_flag))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int c = 0; c < o_cols; c += 16) {
          uint32_t o[16], w[16];
          tmem_get16(tmem_o + lanes + (uint32_t)(o_first + c), o);
#pragma unroll
          for (int e = 0; e < 16; ++e) w[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
          tmem_st16(tmem_o + lanes + (uint32_t)(o_first + c), w);
        }
        l *= corr;
      }
      const float ref = m == -INFINITY ? 0.f : m;
      float sum = 0.f;
      uint32_t p[16];
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        const __nv_bfloat162 w = __floats2bfloat162_rn(fast_exp2(v[e] - ref), fast_exp2(v[e + 1] - ref));
        const float2 b = __bfloat1622float2(w);
        sum += b.x + b.y;
        p[e >> 1] = *reinterpret_cast<const uint32_t*>(&w);
      }
      l += sum;
      tmem_st16(t_s + 16u * half, p);
      if (j0 + KB - 1 > last_pos || (j0 < lo_min && j0 + KB > kept)) {      // keys that no row sees
        Mark at = v_at;
        for (int c = 0; c < a.v_chunks && ok; ++c) {
          ok = mbar_wait_warp(&sm.full[at.slot], at.ph, abort_flag);
          for (int e = threadIdx.x; e < KB * 8; e += SOFT_THREADS) {
            const int j = j0 + (e >> 3);
            if (j > last_pos || (j < lo_min && j >= kept))
              *reinterpret_cast<uint4*>(ring + at.slot * SLOT + e * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          at.step(1, a.slots);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!ok) break;
      }
      v_at.step(per_block, a.slots);
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.p_full[i & 1]);
    }
    // (S of the last block says that P V of the last but two is done: a parity tells one block from the next, not two)
    if (ok && n_blocks > 1) ok = mbar_wait_warp(&sm.o_full, (uint32_t)(n_blocks & 1), abort_flag);
    if (ok) ok = mbar_wait_warp(&sm.o_full, (uint32_t)((n_blocks - 1) & 1), abort_flag);
    if (ok) {
      sm.row_max[n_blocks & 1][half][r] = l;
      __syncwarp();
      if (lane == 0) mbar_arrive(x_full);
      ok = mbar_wait_warp(x_full, (uint32_t)(n_blocks & 1), abort_flag);
    }
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      l = sm.row_max[n_blocks & 1][0][r] + sm.row_max[n_blocks & 1][1][r];
      const int h = h0 + (r & (HG - 1));
      const __nv_bfloat16* gate = tq < nq ? after_wait(a.gate) : nullptr;
      float f = l > 0.f ? 1.f / l : 0.f;
      if (gate != nullptr) {
        gate += (size_t)(t0 + tq) * a.ldg + (a.gate_cols ? (size_t)h * a.Dv : (size_t)h);
        if (!a.gate_cols) f *= 1.f / (1.f + expf(-__bfloat162float(gate[0])));
      }
      TO* out = reinterpret_cast<TO*>(a.out);
      uint4* stg = reinterpret_cast<uint4*>(s_hi) + warp * 128;      // the queries are done with
      constexpr int PER = 16 / sizeof(TO), ROUND = 4 * PER;          // columns of a piece, and of the 64 bytes of a row a round
      for (int c = 0; c < o_cols; c += 32) {
        uint32_t o[32];
        tmem_get32(tmem_o + lanes + (uint32_t)(o_first + c), o);
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          float u = __uint_as_float(o[e]) * f;
          const int col = o_first + c + e;
          if (a.gate_cols && gate != nullptr && col < a.Dv) u *= 1.f / (1.f + expf(-__bfloat162float(gate[col])));
          o[e] = __float_as_uint(u);
        }
#pragma unroll
        for (int p0 = 0; p0 < 32; p0 += ROUND) {
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            uint4 u;
            if (sizeof(TO) == 2) {
              float w[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) w[e] = __uint_as_float(o[(8 * p + e) & 31]);
              u = pack8(w);
            } else {
              const int e = (p0 + 4 * p) & 31;
              u = make_uint4(o[e], o[e + 1], o[e + 2], o[e + 3]);
            }
            stg[stage_index(lane, p)] = u;
          }
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 4; ++j) {      // four lanes on a row's 64 bytes
            const int rw = 8 * j + (lane >> 2), rr = (warp & 3) * 32 + rw, piece = lane & 3;
            const uint4 u = stg[stage_index(rw, piece)];
            const int col = o_first + c + p0 + piece * PER;
            if ((rr >> hg_shift) >= nq || col >= a.Dv) continue;
            TO* dst = out + (size_t)(t0 + (rr >> hg_shift)) * a.ldo + (size_t)(h0 + (rr & (HG - 1))) * a.ohs + col;
            if (a.vec_out) {                 // Dv is a multiple of 8: a piece lies inside as a whole
              *reinterpret_cast<uint4*>(dst) = u;
            } else {
              const TO* w = reinterpret_cast<const TO*>(&u);
#pragma unroll
              for (int e = 0; e < PER; ++e) dst[e] = w[e];
            }
          }
          __syncwarp();
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  const bool aborted = sm.abort_flag != 0;
  if (threadIdx.x == 0 && aborted) atomicOr(a.status, MLXB_ST_WAIT_TIMEOUT);
  if (warp == MMA_WARP) {
    if (aborted && elect_one()) {      // products in flight may still use the tensor memory that is freed below
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
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"(a.tmem_cols) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------- host side

// How a launch is laid out, or false where the sizes are not served.
struct Plan { int HG, steps, chunks, v_chunks, lo_tmem, slots, tmem_cols; size_t smem; };
static bool plan_of(int Hq, int Hkv, int Hv, int Dk, int Dv, int krs, int vrs, int page, int talk, int shared_v, Plan* p) {
  if (Hq <= 0 || Hkv <= 0 || Hv <= 0 || Hq % Hkv || Hkv % Hv || Dk <= 0 || Dk % 4 || Dv <= 0 || Dv % 8 || krs % 8 || vrs % 8) return false;
  if (page < 8 || page > KB || (page & (page - 1))) return false;
  if (talk && (Dk % 64 || krs != Dk)) return false;                // a chunk of 64 columns lies in one key head
  if (shared_v && (Hv != Hkv || talk || vrs != krs || Dv > Dk)) return false;
  const int rep = Hq / Hkv;
  const int width = talk ? Dk * Hkv : Dk;
  p->steps = (width + 15) / 16;
  if (!talk && 16 * p->steps > (krs + 15) / 16 * 16) return false;
  p->chunks = (p->steps + 3) / 4;
  p->v_chunks = (Dv + 63) / 64;
  int hg = 1;
  while (hg * 2 <= M && rep % (hg * 2) == 0) hg *= 2;
  p->HG = hg;
  const int left = 512 - 2 * KB - 64 * p->v_chunks;                // columns of tensor memory for the low halves
  if (left < 0) return false;
  p->lo_tmem = left / 32 < p->chunks ? left / 32 : p->chunks;
  const int cols = 2 * KB + 32 * p->lo_tmem + 64 * p->v_chunks;
  p->tmem_cols = cols <= 256 ? 256 : 512;
  const long long queries = (long long)(2 * p->chunks - p->lo_tmem) * Q_CHUNK, most = 226 * 1024 - (long long)sizeof(Control) - 1024;
  if (queries >= most) return false;
  const long long slots = (most - queries) / SLOT;
  p->slots = slots < MAX_SLOTS ? (int)slots : MAX_SLOTS;
  // S of a block runs while the block before still has its values in the ring
  const int need = shared_v ? 2 * p->chunks : p->chunks + 2 * p->v_chunks;
  if (p->slots < need || p->slots < 2) return false;
  p->smem = (size_t)(queries + (long long)p->slots * SLOT + (long long)sizeof(Control) + 1024);
  return true;
}

MLXB_EXPORT int mlxb_attention_wide_tcgen05_supported(int Hq, int Hkv, int Hv, int Dk, int Dv, int krs, int vrs, int page, int talk,
                                                      int shared_v) {
  Plan p;
  return plan_of(Hq, Hkv, Hv, Dk, Dv, krs, vrs, page, talk, shared_v, &p) ? 1 : 0;
}

static int make_map(CUtensorMap* map, const void* base, long long rows, int cols, int box_rows, const char* what) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * sizeof(__nv_bfloat16)};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    const char* msg = nullptr;
    cuGetErrorString(r, &msg);
    return mlxb_fail(MLXB_BAD_ARG, "attention (wide, tcgen05): tensor map of %s (%lld x %d): %s", what, rows, cols, msg ? msg : "?");
  }
  return 0;
}

// The arguments of mlxb_attention_wide_tc without those of single rows.  q: 16-byte rows (ldq, qhs multiples of 4).
MLXB_EXPORT int mlxb_attention_wide_tcgen05(int out_f32, const float* q, int ldq, int qhs, const int* tiles, int n_tiles, int tile_q,
                                            const int* block_table, int max_pages, int n_pages, int page, int Hq, int Hkv, int Dk,
                                            int Dv, int krs, int vrs, int window, int chunk, float scale, const float* talk,
                                            const void* k_pool, const void* v_pool, const void* gate, int ldg, void* out, int ldo,
                                            int ohs, int* status, float softcap, int keep_first, int gate_cols, int Hv,
                                            cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  if (Hv <= 0) Hv = Hkv;
  Plan p;
  const int shared_v = v_pool == k_pool;
  if (!plan_of(Hq, Hkv, Hv, Dk, Dv, krs, vrs, page, talk != nullptr, shared_v, &p) || tile_q <= 0 || qhs < Dk || ohs < Dv || (ldq & 3) ||
      (qhs & 3) || (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) || Hq / p.HG > 65535)
    return mlxb_fail(MLXB_BAD_ARG, "attention (wide, tcgen05): %d/%d heads, sizes %d/%d in rows of %d/%d, page %d", Hq, Hkv, Dk, Dv, krs,
                     vrs, page);
  CUtensorMap mk, mv;
  if (int e = make_map(&mk, k_pool, (long long)n_pages * Hkv * page, krs, page, "k pool")) return e;
  if (int e = make_map(&mv, v_pool, (long long)n_pages * Hv * page, vrs, page, "v pool")) return e;
  const int TQ = M / p.HG, subs = (tile_q + TQ - 1) / TQ, size = out_f32 ? 4 : 2;
  WideArgs a = {};
  a.q = q; a.tiles = tiles; a.block_table = block_table; a.talk = talk; a.gate = (const __nv_bfloat16*)gate; a.out = out; a.status = status;
  a.ldq = ldq; a.qhs = qhs; a.subs = subs; a.n_tiles = n_tiles; a.max_pages = max_pages; a.n_pages = n_pages; a.page = page;
  a.Hq = Hq; a.Hkv = Hkv; a.Hv = Hv; a.Dk = Dk; a.Dv = Dv; a.window = window; a.chunk = chunk; a.ldg = ldg; a.ldo = ldo; a.ohs = ohs;
  a.keep_first = window > 0 ? keep_first : 0;                      // without a window every earlier position is visible anyway
  a.gate_cols = gate_cols;
  a.HG = p.HG; a.steps = p.steps; a.chunks = p.chunks; a.v_chunks = p.v_chunks; a.lo_tmem = p.lo_tmem; a.slots = p.slots;
  a.shared_v = shared_v; a.tmem_cols = p.tmem_cols;
  a.vec_out = ((uintptr_t)out & 15) == 0 && (long long)ldo * size % 16 == 0 && (long long)ohs * size % 16 == 0;
  a.mix_fast = talk != nullptr && Hq / Hkv <= 4 && p.HG * Hq <= MAX_MIX;
  a.scale = scale; a.softcap = softcap;
  const dim3 grid((unsigned)n_tiles * subs, Hq / p.HG);
  static SharedLimit limits[2];
  auto go = [&](auto kernel, SharedLimit& limit) {
    const cudaError_t e = limit.raise(kernel, 226 * 1024);
    if (e != cudaSuccess)
      return mlxb_fail((int)e, "attention (wide, tcgen05): %zu bytes of shared memory: %s", p.smem, cudaGetErrorString(e));
    launch_pdl(kernel, grid, dim3(THREADS), p.smem, stream, mk, mv, a);
    return mlxb_check_launch("attention (wide, tcgen05)");
  };
  if (out_f32) return go(attention_wide_tcgen05_kernel<float>, limits[0]);
  return go(attention_wide_tcgen05_kernel<__nv_bfloat16>, limits[1]);
}
