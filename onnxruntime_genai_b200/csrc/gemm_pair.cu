// Linear layers of prompt-sized steps on pairs of SMs:  C[M,N] = A[M,K] * W[N,K]^T  (+ epilogue)  with bf16 weights, packed int4 block-32
// weights (records of gemm_w4.cu) or packed MXFP4 experts (records and tile list of gemm_fp4.cu).
//
// A cluster of two CTAs walks a list of output tiles of 256 weight rows x up to 256 tokens (`tcgen05.mma.cta_group::2`, M = 256): each CTA
// holds 128 of the weight rows and HALF of the token rows in its shared memory and the accumulator of its own 128 rows in its tensor memory,
// so a k-block of 64 brings 32 KiB (packed weights: 21 KiB) into an SM for 512 cycles of MMAs where one CTA per 128 x 256 tile needs 48 KiB.
//
// A stage holds TWO k-blocks (K = 128).  A role's pass over a stage costs 350 to 700 cycles of dependent instructions (wait, vote, election, copies
// or MMAs) whatever the tile, which with stages of one k-block was more than its MMAs take: 305 ns per k-block for any tile of 32 to 256 tokens, now
// 155 (32 .. 128 tokens) to 280 (256 tokens).
//
// Warps of a CTA: 0 copies, 1 issues the MMAs (of the cluster's first CTA), both as whole warps with one elected lane; 2..5 drain accumulators (two
// of 256 columns in tensor memory, so that a tile is drained under the next one's main loop; 32 token columns at a time through a staging tile that
// turns a weight row per thread into 16-byte row segments); 6 copies packed records, 7.. expand them into the swizzled weight tiles (two teams of
// eight warps that take every other stage; a thread expands one weight row of one k-block).
// Copies of both CTAs are counted on the FIRST CTA's barrier of a stage; a commit frees the stage in both CTAs.  The number of token
// tiles is chosen by the launcher (PlanPair).  All waits are bounded; after a failed one every role leaves its loop, both CTAs meet
// at the last cluster barrier and return with the status word set.
//
// Measured (us, before: one CTA per 128 x 256 tile; TFLOP/s now): M 4096, N 28672, K 4096 667 -> 630 (1528); M 4096, N 4096, K 4096 106 -> 93 (1476); M 806,
// N 6144, K 4096 54 -> 35 (1147).  int4: M 777, N 16384, K 3072 174 -> 79 (987), M 2500 433 -> 194 (1298).  MXFP4, 32 experts of 5760 x 2880, 6000 rows: 389 -> 189.
#include <cstdlib>

#include "gemm_common.cuh"
#include "kernels.h"
#include "packed_weights.cuh"

namespace ogb {

enum PairWeights : int { PAIR_BF16 = 0, PAIR_W4 = 1, PAIR_FP4_F16 = 2, PAIR_FP4_BF16 = 3 };

constexpr int PAIR_MAX_BT = 256;                                   // tokens of a tile
constexpr int PAIR_KB = 2;                                         // k-blocks of a stage
constexpr int PAIR_A_TILE = PAIR_MAX_BT / 2 * GEMM_BLOCK_K * 2;    // a CTA's half of the token rows of a k-block, 16 KiB
constexpr int PAIR_STAGING_LD = GEMM_BLOCK_N + 4;                  // floats of a token column in the staging tile
constexpr int PAIR_STAGING_BYTES = 32 * PAIR_STAGING_LD * 4;

template <int FMT>
struct PairCfg {
  static constexpr bool PACKED = FMT != PAIR_BF16;
  static constexpr int A_STAGES = 3;
  static constexpr int W_STAGES = PACKED ? 2 : A_STAGES;            // weight tiles (bf16: part of the stage)
  static constexpr int RAW = PACKED ? 4 : 0;                        // stages of packed records in flight
  static constexpr int REC_BYTES = FMT == PAIR_W4 ? W4_RECORD_BYTES : FP4_RECORD_BYTES;
  static constexpr int TEAMS = 2;                                   // teams of eight expanding warps
  static constexpr int THREADS = GEMM_THREADS + (PACKED ? 32 + TEAMS * 256 : 0);
  static constexpr int W_OFF = A_STAGES * PAIR_KB * PAIR_A_TILE;
  static constexpr int RAW_OFF = W_OFF + W_STAGES * PAIR_KB * W_TILE_BYTES;
  static constexpr int STAGING_OFF = RAW_OFF + RAW * PAIR_KB * REC_BYTES;
  static constexpr int BAR_OFF = STAGING_OFF + PAIR_STAGING_BYTES;
  static constexpr int SMEM_BYTES = BAR_OFF + 512 + 1024;           // + barriers, + alignment slack
  static_assert(RAW_OFF % 1024 == 0 && STAGING_OFF % 16 == 0 && BAR_OFF % 8 == 0, "alignment");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of an SM");
};

struct PairArgs {
  int bt;               // tokens of a tile: a multiple of 32 up to 256 (grouped: of the list's tiles)
  int m_tiles;          // token tiles (grouped: from the list)
  int n_pairs;          // tiles of 256 weight rows
  int a_box;            // token rows of one copy: half a tile
  const uint8_t* packed;
  int n_tiles;          // record tiles of 128 weight rows per k-block
};

// ------------------------------------------------------------------------------- pair forms of the PTX wrappers
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// into this CTA's shared memory, counted on the barrier at the cluster address `bar`
__device__ __forceinline__ void pair_tma_load_2d(void* smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void pair_umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at this offset in both CTAs once every MMA issued so far is done
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(uint16_t(3)) : "memory");
}
// bar: cluster address.  The arrival names no scope, so what PTX promises is a release to the arriving CTA, while the waiter of the second CTA's arrivals is in
// the first one: the text of the memory model does not order them.  What this rests on: the data concerned are the arriving CTA's own shared memory, whose
// writers have each passed the proxy fence (which completes their stores) before their warp arrives, and its tensor memory, whose reads are complete after
// tcgen05.wait; no cache lies between them and the tensor core that the arrival releases.  Arrivals of the scope of the cluster, all of them or relayed by one
// warp of the second CTA, would be ordered by the text too and cost (us, none / all / relayed): int4 777 tokens, N 16384, K 3072 77 / 115 / 107,
// MXFP4 6000 rows of 32 experts, 5760 x 2880 178 / 277 / 266.
__device__ __forceinline__ void cluster_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool cluster_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// mbar_wait_bounded for barriers on which the other CTA arrives
__device__ __forceinline__ bool cluster_wait_bounded(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint64_t timeout_ns = 2000000000ull) {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (!cluster_try_wait(bar, parity)) {
    if ((++spins & 0x3ff) == 0) {
      if (*abort_flag) return false;
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > timeout_ns) return false;
    }
  }
  return true;
}

// v: the accumulators (+ bias) of eight weight rows, u: (paired) of the up rows 64 further
__device__ __forceinline__ void pair_activate8(const GemmParams& p, float (&v)[8], const float (&u)[8]) {
  if (p.act_pair == 1) {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = silu(v[q]) * u[q];
  } else if (p.act_pair == 3) {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = fmaxf(v[q], 0.f) * u[q];
  } else if (p.act_pair == 4) {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = gelu_tanh(v[q]) * u[q];
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float g = p.act_limit > 0.f ? fminf(v[q], p.act_limit) : v[q];
      const float w = p.act_limit > 0.f ? fminf(fmaxf(u[q], -p.act_limit), p.act_limit) : u[q];
      v[q] = g / (1.f + __expf(-p.act_alpha * g)) * (w + 1.f);
    }
  }
}
// Eight columns of a row: residual and store.  whole: all eight exist and every row segment is aligned for 16-byte accesses.
__device__ __forceinline__ void pair_store8(const StoreArgs& a, int m, int col, bool whole, float (&v)[8]) {
  if (!whole || a.out_kind == 2) {
    epi_store8(a, m, col, make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]));
    return;
  }
  if (a.residual) {
    if (a.res_fp32) {
      const float4* r = reinterpret_cast<const float4*>(static_cast<const float*>(a.residual) + size_t(m) * a.ldr + col);
      const float4 x = r[0], y = r[1];
      v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w; v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
    } else {
      const uint4 q = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.residual) + size_t(m) * a.ldr + col);
      const float2 x0 = unpack_bf16x2(q.x), x1 = unpack_bf16x2(q.y), x2 = unpack_bf16x2(q.z), x3 = unpack_bf16x2(q.w);
      v[0] += x0.x; v[1] += x0.y; v[2] += x1.x; v[3] += x1.y; v[4] += x2.x; v[5] += x2.y; v[6] += x3.x; v[7] += x3.y;
    }
  }
  if (a.out_kind == 1) {
    float4* dst = reinterpret_cast<float4*>(static_cast<float*>(a.C) + size_t(m) * a.ldc + col);
    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.C) + size_t(m) * a.ldc + col) =
        make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
  }
}

template <int FMT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<FMT>::THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, const GemmParams p, const PairArgs a) {
  using Cfg = PairCfg<FMT>;
  constexpr bool PACKED = Cfg::PACKED;
  constexpr int AS = Cfg::A_STAGES, WS = Cfg::W_STAGES, RAW = Cfg::RAW > 0 ? Cfg::RAW : 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* staging = reinterpret_cast<float*>(smem + Cfg::STAGING_OFF);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);   // [AS] copies -> MMA (first CTA's)
  uint64_t* empty = full + AS;                                          // [AS] MMA -> copies (both)
  uint64_t* acc_full = empty + AS;                                      // [2] MMA -> drain (both)
  uint64_t* acc_empty = acc_full + 2;                                   // [2] drain of both CTAs -> MMA (first CTA's)
  uint64_t* deq_full = acc_empty + 2;                                   // [WS] expanded in both CTAs -> MMA (first CTA's)
  uint64_t* w_empty = deq_full + WS;                                    // [WS] MMA -> expanders (both)
  uint64_t* raw_full = w_empty + WS;                                    // [RAW] local
  uint64_t* raw_empty = raw_full + RAW;                                 // [RAW] local
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(raw_empty + RAW);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* epi_abort = reinterpret_cast<volatile int*>(tmem_slot + 2);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
  const int num_kb = p.total_kb, num_st = (num_kb + PAIR_KB - 1) / PAIR_KB;      // (the last stage of a tile may hold one k-block)
  const bool grouped = p.grp.tile_expert != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < AS; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
    if (PACKED) {
      for (int s = 0; s < WS; ++s) { mbar_init(&deq_full[s], 16); mbar_init(&w_empty[s], 1); }
      for (int s = 0; s < RAW; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 8); }
    }
    *abort_flag = 0;
    *epi_abort = 0;
    mbar_fence_init();
    if (!PACKED) tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
  }
  __syncwarp();
  if (warp == 2) pair_tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  cluster_sync_all();                      // barriers of both CTAs are initialised, tensor memory is allocated
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (p.pdl) pdl_launch_dependents();
  if (grouped && p.pdl) pdl_wait();        // the tile list is written by the kernel before this one
  const int m_tiles = grouped ? *p.grp.num_tiles : a.m_tiles;
  const int total_tiles = m_tiles * a.n_pairs;
  // Tiles that run at the same time share operands in L2: the few weight tiles of the moment and all tokens, or (experts, whose tiles
  // of one expert are neighbours in the list) the tokens of a few experts and their weights.
  struct Tile { int n_tile, row0, rows, expert; };
  auto tile_at = [&](int t) {
    Tile x;
    if (grouped) {
      const int m = t / a.n_pairs;
      x.n_tile = (t - m * a.n_pairs) * 2 + int(rank);
      x.row0 = p.grp.tile_row0[m]; x.rows = p.grp.tile_rows[m]; x.expert = p.grp.tile_expert[m];
    } else {
      const int n = t / m_tiles;
      x.n_tile = n * 2 + int(rank);
      x.row0 = (t - n * m_tiles) * a.bt; x.rows = min(a.bt, p.M - x.row0); x.expert = 0;
    }
    return x;
  };
  auto cols_of = [&](int rows) { return min(a.bt, (rows + 31) & ~31); };     // token columns of the MMA
  auto fail = [&](int code) { atomicMax(p.status, code); *abort_flag = 1; };
  auto stage_a = [&](int s) { return smem + s * (PAIR_KB * PAIR_A_TILE); };
  auto stage_w = [&](int s) { return smem + Cfg::W_OFF + s * (PAIR_KB * W_TILE_BYTES); };

  if (warp == 0) {
    // ------------------------------------------------------------------ copies: k-blocks of all tiles, back to back
    bool waited = grouped || !p.pdl, ok = true;
    int it = 0, s = 0;                                                 // stages filled so far, the next one
    uint32_t ph = 1;
    for (int t = first; t < total_tiles && ok; t += step) {
      const Tile x = tile_at(t);
      // One copy brings half of a whole tile's rows, of which a tile that ends early uses the first ones.  (The loop over `copies` runs once; as straight-line
      // code the kernel is slower: packed weights 1.5 to 3 %, bf16 2 %, the geometric mean of 84 sizes, with the same registers.)
      const int half = cols_of(x.rows) >> 1, copies = (half + a.a_box - 1) / a.a_box;
      const uint32_t bytes = uint32_t(copies * a.a_box * GEMM_BLOCK_K * 2 + (PACKED ? 0 : W_TILE_BYTES));
      const int row = x.row0 + int(rank) * half, w_row = x.n_tile * GEMM_BLOCK_N;
      for (int i = 0; i < num_st; ++i) {
        const int nk = min(PAIR_KB, num_kb - i * PAIR_KB), k0 = i * (PAIR_KB * GEMM_BLOCK_K);
        if (it >= AS) ok = __all_sync(0xffffffffu, cluster_wait_bounded(&empty[s], ph, abort_flag));
        if (!ok) { fail(OGB_ERR_WAIT_TMA); break; }
        const uint32_t bar = dsmem_addr(smem_u32(&full[s]), 0);
        const bool early = !waited;      // the first weight tiles may go out before the previous kernel has finished; tokens may not
        if (early) {
          if (elect_one()) {
            if (rank == 0) mbar_expect_tx(&full[s], 2 * nk * bytes);
            if (!PACKED) for (int h = 0; h < nk; ++h) pair_tma_load_2d(stage_w(s) + h * W_TILE_BYTES, &tmap_w, bar, k0 + h * GEMM_BLOCK_K, w_row);
          }
          __syncwarp();
          pdl_wait();
          waited = true;
        }
        if (elect_one()) {
          if (rank == 0 && !early) mbar_expect_tx(&full[s], 2 * nk * bytes);
#pragma unroll
          for (int h = 0; h < PAIR_KB; ++h) {
            if (h >= nk) break;
            if (!PACKED && !early) pair_tma_load_2d(stage_w(s) + h * W_TILE_BYTES, &tmap_w, bar, k0 + h * GEMM_BLOCK_K, w_row);
            for (int c = 0; c < copies; ++c)
              pair_tma_load_2d(stage_a(s) + h * PAIR_A_TILE + c * a.a_box * 128, &tmap_a, bar, k0 + h * GEMM_BLOCK_K, row + c * a.a_box);
          }
        }
        __syncwarp();
        ++it;
        if (++s == AS) { s = 0; ph ^= 1; }
      }
    }
    if (!ok) {   // copies already issued still write the pair's shared memory: give them time to land
      volatile int never = 0;
      if (rank == 0) for (int i = max(0, it - AS); i < it; ++i) mbar_wait_bounded(&full[i % AS], (i / AS) & 1, &never, 200000000ull);
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ------------------------------------------------------------------ MMAs of the pair: alternate the two accumulators
      int s = 0, ws = 0, j = 0;
      uint32_t ph = 0, wph = 0;
      bool ok = true;
      for (int t = first; t < total_tiles && ok; t += step, ++j) {
        const int buf = j & 1;
        if (j >= 2) ok = __all_sync(0xffffffffu, cluster_wait_bounded(&acc_empty[buf], ((j >> 1) & 1) ^ 1, abort_flag));
        if (!ok) { fail(OGB_ERR_WAIT_MMA); break; }
        tc_fence_after();
        const uint32_t acc = tmem_base + uint32_t(buf * PAIR_MAX_BT);
        const uint32_t idesc = umma_idesc_f16(2 * GEMM_BLOCK_N, cols_of(tile_at(t).rows), FMT == PAIR_FP4_F16 ? 0 : 1);
        for (int i = 0; i < num_st; ++i) {
          bool got = true;
          if (PACKED) got = cluster_wait_bounded(&deq_full[ws], wph, abort_flag);
          got = got && cluster_wait_bounded(&full[s], ph, abort_flag);
          if (!__all_sync(0xffffffffu, got)) { fail(OGB_ERR_WAIT_TMA); ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            const uint64_t dw = umma_desc_sw128(smem_u32(stage_w(ws))), db = umma_desc_sw128(smem_u32(stage_a(s)));
            const int nk = min(PAIR_KB, num_kb - i * PAIR_KB);
#pragma unroll
            for (int h = 0; h < PAIR_KB; ++h) {
              if (h >= nk) break;
#pragma unroll
              for (int k = 0; k < GEMM_BLOCK_K / GEMM_UMMA_K; ++k)
                pair_umma_f16(acc, dw + (h * W_TILE_BYTES + k * GEMM_UMMA_K * 2) / 16, db + (h * PAIR_A_TILE + k * GEMM_UMMA_K * 2) / 16, idesc,
                              (i > 0 || h > 0 || k > 0) ? 1u : 0u);
            }
            pair_commit(&empty[s]);
            if (PACKED) pair_commit(&w_empty[ws]);
            if (i == num_st - 1) pair_commit(&acc_full[buf]);
          }
          __syncwarp();
          if (++s == AS) { s = 0; ph ^= 1; }
          if (++ws == WS) { ws = 0; wph ^= 1; }
        }
      }
    }
  } else if (warp < 6) {
    // -------------------------------------------------------------------- drain: warps 2..5
    const int et = threadIdx.x - 64;
    const int quarter = warp & 3;            // TMEM lanes this warp may read
    const int row = quarter * 32 + lane;     // weight row of the tile held by this thread
    const bool pair = p.act_pair != 0;
    const StoreArgs sa{p.C, p.residual, p.ldc, p.ldr, p.out_fp32, pair ? p.N / 2 : p.N, p.res_fp32};
    const int out_size = p.out_fp32 == 1 ? 4 : 2, res_size = p.res_fp32 ? 4 : 2;
    const bool aligned = ((reinterpret_cast<uintptr_t>(p.C) | size_t(p.ldc) * out_size) & 15) == 0 &&
                         (!p.residual || ((reinterpret_cast<uintptr_t>(p.residual) | size_t(p.ldr) * res_size) & 15) == 0);
    // the eight columns of a token row that this thread finishes: plain, of its own warp's rows; paired, of the 64 gate rows
    const int seg = pair ? (et & 7) * 8 : quarter * 32 + (lane & 3) * 8;
    const int tok = pair ? et >> 3 : lane >> 2;
    if (p.pdl) pdl_wait();                   // residual reads and all stores come after the previous kernel
    int j = 0;
    for (int t = first; t < total_tiles; t += step, ++j) {
      const int buf = j & 1;
      const Tile x = tile_at(t);
      // a failed wait is published in a word only these threads write, before the barrier: all 128 take the same branch
      if (!cluster_wait_bounded(&acc_full[buf], (j >> 1) & 1, abort_flag, 4000000000ull)) { fail(OGB_ERR_WAIT_MMA); *epi_abort = 1; }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (*epi_abort) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(buf * PAIR_MAX_BT);
      const int n0 = x.n_tile * GEMM_BLOCK_N, rows = n0 < p.N ? x.rows : 0;
      const int col = x.n_tile * (pair ? 64 : GEMM_BLOCK_N) + seg;
      const bool whole = aligned && col + 8 <= sa.n_out;
      float b0[8], b1[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        b0[q] = p.bias && n0 + seg + q < p.N ? bf2f(p.bias[size_t(x.expert) * p.N + n0 + seg + q]) : 0.f;
        b1[q] = p.bias && pair && n0 + seg + 64 + q < p.N ? bf2f(p.bias[size_t(x.expert) * p.N + n0 + seg + 64 + q]) : 0.f;
      }
      for (int c0 = 0; c0 < rows; c0 += 32) {
        uint32_t r0[16], r1[16];
        __syncwarp();
        tmem_ld16(taddr + c0, r0);
        tmem_ld16(taddr + c0 + 16, r1);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          staging[q * PAIR_STAGING_LD + row] = __uint_as_float(r0[q]);
          staging[(q + 16) * PAIR_STAGING_LD + row] = __uint_as_float(r1[q]);
        }
        // all values of the chunk are read before the first store: a store through a generic pointer would order the reads behind it
        if (pair) {
          asm volatile("bar.sync 1, 128;" ::: "memory");
          float4 g[2][2], h[2][2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float4* src = reinterpret_cast<const float4*>(staging + (tok + k * 16) * PAIR_STAGING_LD + seg);
            g[k][0] = src[0]; g[k][1] = src[1]; h[k][0] = src[16]; h[k][1] = src[17];
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int mc = c0 + tok + k * 16;
            float v[8] = {g[k][0].x + b0[0], g[k][0].y + b0[1], g[k][0].z + b0[2], g[k][0].w + b0[3], g[k][1].x + b0[4], g[k][1].y + b0[5], g[k][1].z + b0[6], g[k][1].w + b0[7]};
            const float u[8] = {h[k][0].x + b1[0], h[k][0].y + b1[1], h[k][0].z + b1[2], h[k][0].w + b1[3], h[k][1].x + b1[4], h[k][1].y + b1[5], h[k][1].z + b1[6], h[k][1].w + b1[7]};
            pair_activate8(p, v, u);
            if (mc < rows && col < sa.n_out) pair_store8(sa, x.row0 + mc, col, whole, v);
          }
        } else {
          __syncwarp();
          float4 g[4][2];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4* src = reinterpret_cast<const float4*>(staging + (tok + k * 8) * PAIR_STAGING_LD + seg);
            g[k][0] = src[0]; g[k][1] = src[1];
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int mc = c0 + tok + k * 8;
            float v[8] = {g[k][0].x + b0[0], g[k][0].y + b0[1], g[k][0].z + b0[2], g[k][0].w + b0[3], g[k][1].x + b0[4], g[k][1].y + b0[5], g[k][1].z + b0[6], g[k][1].w + b0[7]};
            if (p.act_one) epi_act8(p.act_one, v);
            if (mc < rows && col < sa.n_out) pair_store8(sa, x.row0 + mc, col, whole, v);
          }
        }
      }
      // accumulator drained: hand it back to the MMA warp of the pair
      tc_fence_before();
      __syncwarp();
      if (lane == 0) cluster_arrive(dsmem_addr(smem_u32(&acc_empty[buf]), 0));
    }
  } else if constexpr (PACKED) {
    if (warp == 6) {
      // ------------------------------------------------------------------ packed records (nothing earlier in the stream writes them: no wait)
      bool ok = true;
      int it = 0, s = 0;
      uint32_t ph = 1;
      const size_t rec_stride = size_t(a.n_tiles) * Cfg::REC_BYTES;
      for (int t = first; t < total_tiles && ok; t += step) {
        const Tile x = tile_at(t);
        const int nt = min(x.n_tile, a.n_tiles - 1);                        // past the last tile: any record, the result is not stored
        const uint8_t* src = a.packed + (size_t(x.expert) * num_kb * a.n_tiles + nt) * Cfg::REC_BYTES;
        for (int i = 0; i < num_st; ++i, src += PAIR_KB * rec_stride) {
          if (it >= RAW) ok = __all_sync(0xffffffffu, cluster_wait_bounded(&raw_empty[s], ph, abort_flag));
          if (!ok) { fail(OGB_ERR_WAIT_TMA); break; }
          if (elect_one()) {
            const int nk = min(PAIR_KB, num_kb - i * PAIR_KB);
            mbar_expect_tx(&raw_full[s], nk * Cfg::REC_BYTES);
            uint8_t* dst = smem + Cfg::RAW_OFF + s * (PAIR_KB * Cfg::REC_BYTES);
#pragma unroll
            for (int h = 0; h < PAIR_KB; ++h) if (h < nk) bulk_copy_g2s(dst + h * Cfg::REC_BYTES, src + h * rec_stride, Cfg::REC_BYTES, &raw_full[s]);
          }
          __syncwarp();
          ++it;
          if (++s == RAW) { s = 0; ph ^= 1; }
        }
      }
      if (!ok) {   // copies already issued still write shared memory: give them time to land
        volatile int never = 0;
        for (int i = max(0, it - RAW); i < it; ++i) mbar_wait_bounded(&raw_full[i % RAW], (i / RAW) & 1, &never, 200000000ull);
      }
    } else {
      // ------------------------------------------------------------------ expanders: thread = weight row of a k-block
      const int dt = threadIdx.x - GEMM_THREADS - 32, team = dt >> 8, half = (dt >> 7) & 1, row = dt & 127;
      const int my_tiles = first < total_tiles ? (total_tiles - first + step - 1) / step : 0;
      bool ok = true;
      int g = 0;                                                              // stages so far
      for (int j = 0; j < my_tiles && ok; ++j) {
        for (int i = 0; i < num_st; ++i, ++g) {
          if (g % Cfg::TEAMS != team) continue;
          const int ws = g % WS, kb = i * PAIR_KB + half, rs = g % RAW;
          uint4 out[8];
          ok = mbar_wait_bounded(&raw_full[rs], (g / RAW) & 1, abort_flag);
          if (kb < num_kb) {
            const uint8_t* rec = smem + Cfg::RAW_OFF + (rs * PAIR_KB + half) * Cfg::REC_BYTES;
            const uint4 q0 = *reinterpret_cast<const uint4*>(rec + row * 32);
            const uint4 q1 = *reinterpret_cast<const uint4*>(rec + row * 32 + 16);
            const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            if constexpr (FMT == PAIR_W4) {
              const uint2 sz = *reinterpret_cast<const uint2*>(rec + GEMM_BLOCK_N * 32 + row * 8);
              const W4Scale sc[2] = {w4_scale(sz.x), w4_scale(sz.y)};
#pragma unroll
              for (int q = 0; q < 8; ++q) out[q] = deq_w4_word(words[q], sc[q >> 2]);
            } else {
              const uint32_t mul = *reinterpret_cast<const uint16_t*>(rec + GEMM_BLOCK_N * 32 + row * 2);   // exponent fields of the two multipliers
              if constexpr (FMT == PAIR_FP4_F16) {
                // word (q, b) of the record expands to the 16-byte chunk 4 b + q; the stored byte is code + 6, the fp16 field of 2^(code - 127) is code - 112
                const uint32_t s0 = ((mul & 0xFFu) - 118u) * 0x04000400u, s1 = ((mul >> 8) - 118u) * 0x04000400u;
#pragma unroll
                for (int q = 0; q < 8; ++q) out[4 * (q & 1) + (q >> 1)] = deq_fp4_word_f16(words[q], (q & 1) ? s1 : s0);
              } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) out[q] = deq_fp4_word_bf16(words[q], q < 4 ? (mul & 0xFFu) : (mul >> 8));
              }
            }
          }
          if (ok && g >= WS) ok = cluster_wait_bounded(&w_empty[ws], ((g / WS) & 1) ^ 1, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) { fail(OGB_ERR_WAIT_TMA); break; }                          // the warp gives up as one
          if (lane == 0) mbar_arrive(&raw_empty[rs]);                          // every lane has read its row: the vote above
          if (kb < num_kb) {
            uint8_t* dst = stage_w(ws) + half * W_TILE_BYTES + row * 128;
#pragma unroll
            for (int q = 0; q < 8; ++q) *reinterpret_cast<uint4*>(dst + ((q ^ (row & 7)) << 4)) = out[q];
            fence_proxy_async_smem();   // generic-proxy stores -> visible to the tensor core's async proxy
          }
          __syncwarp();
          if (lane == 0) cluster_arrive(dsmem_addr(smem_u32(&deq_full[ws]), 0));
        }
      }
    }
  }

  __syncwarp();
  tc_fence_before();
  cluster_sync_all();      // no CTA leaves while the pair's MMAs, copies or arrivals may still reach its memory
  if (warp == 2) pair_tmem_dealloc(tmem_base, 512);
}

// --------------------------------------------------------------------------------- host side
bool MakeMapBf16(CUtensorMap* out, const void* ptr, int rows, int cols, int ld, int box_rows);  // gemm_tcgen05.cu

template <int FMT>
static int LaunchPair(const CUtensorMap& tw, const CUtensorMap& ta, const GemmParams& p, const PairArgs& a, int clusters, cudaStream_t stream) {
  static bool configured[OGB_MAX_DEVICES] = {};
  if (!set_max_dyn_smem(gemm_pair_kernel<FMT>, PairCfg<FMT>::SMEM_BYTES, configured)) return -3;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(2 * clusters));
  cfg.blockDim = dim3(PairCfg<FMT>::THREADS);
  cfg.dynamicSmemBytes = PairCfg<FMT>::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = p.pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, gemm_pair_kernel<FMT>, tw, ta, p, a) == cudaSuccess ? 0 : -4;
}

static int DevicePairs() {
  static const int n = [] {
    int dev = 0, v = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? v / 2 : 74;
  }();
  return n;
}

// How an [M, N] product is cut into token tiles of equal size (a multiple of 32), and its estimated time: rounds of the pairs x k-blocks x the time of
// a k-block, which is 1.12 ns per token of the tile down to what a role's pass over a stage and the copies' latency take, the drain of the last
// tile and what every launch has.  Measured with weights from HBM, us: M 512, N 28672, K 4096 in 2 / 3 / 4 / 5 tiles 100 / 105 / 121 / 121 (4 / 5 / 7 / 8
// rounds); M 233, N 6144, K 4096 in 1 / 2 / 3 / 4 tiles 27 / 22 / 20 / 32 (1 / 1 / 1 / 2 rounds); M 512, N 4096, K 14336 in 2 / 4 tiles 76 / 63 (1 round).
struct PairPlan { int bt, m_tiles; double ns; };
static PairPlan PlanPair(int M, int N, int total_kb, int pairs, double floor_ns, int force_tiles) {
  const int n_pairs = (N + 255) / 256, least = (M + PAIR_MAX_BT - 1) / PAIR_MAX_BT;
  PairPlan best{0, 0, 0};
  for (int m = force_tiles > 0 ? force_tiles : least; m <= (force_tiles > 0 ? force_tiles : least + 8); ++m) {
    const int bt = min(PAIR_MAX_BT, ((M + m - 1) / m + 31) / 32 * 32), mt = (M + bt - 1) / bt;
    const double rounds = double((n_pairs * mt + pairs - 1) / pairs);
    const double ns = rounds * total_kb * (1.12 * bt > floor_ns ? 1.12 * bt : floor_ns) + bt / 32 * 400.0 + 5000.0;
    if (best.bt == 0 || ns < best.ns) best = {bt, mt, ns};
    if (bt == 32) break;
  }
  return best;
}
constexpr double PAIR_BF16_FLOOR_NS = 200, PAIR_PACKED_FLOOR_NS = 310;

// Estimated times of the paired kernels in ns, to be compared with the other kernels' (gemm_tcgen05.cu, gemm_w4.cu)
double PairBf16Ns(int M, int N, int total_kb) { return PlanPair(M, N, total_kb, DevicePairs(), PAIR_BF16_FLOOR_NS, 0).ns; }
double PairW4Ns(int M, int N, int total_kb) { return PlanPair(M, N, total_kb, DevicePairs(), PAIR_PACKED_FLOOR_NS, 0).ns; }

// force_tiles > 0: that many token tiles instead of the planned number
int LaunchPairBf16(const void* A, int lda, const void* W, int ldw, const GemmParams& p, int force_tiles, cudaStream_t stream) {
  const PairPlan plan = PlanPair(p.M, p.N, p.total_kb, DevicePairs(), PAIR_BF16_FLOOR_NS, force_tiles);
  PairArgs a = {};
  a.n_pairs = (p.N + 255) / 256;
  a.bt = plan.bt;
  a.m_tiles = plan.m_tiles;
  a.a_box = a.bt / 2;
  CUtensorMap tw, ta;
  if (!MakeMapBf16(&tw, W, p.N, p.K, ldw, GEMM_BLOCK_N) || !MakeMapBf16(&ta, A, p.M, p.K, lda, a.a_box)) return -2;
  return LaunchPair<PAIR_BF16>(tw, ta, p, a, min(DevicePairs(), a.n_pairs * a.m_tiles), stream);
}

int LaunchPairW4(const void* A, int lda, const uint8_t* packed, const GemmParams& p, int force_tiles, cudaStream_t stream) {
  const PairPlan plan = PlanPair(p.M, p.N, p.total_kb, DevicePairs(), PAIR_PACKED_FLOOR_NS, force_tiles);
  PairArgs a = {};
  a.n_pairs = (p.N + 255) / 256;
  a.bt = plan.bt;
  a.m_tiles = plan.m_tiles;
  a.a_box = a.bt / 2;
  a.packed = packed;
  a.n_tiles = (p.N + GEMM_BLOCK_N - 1) / GEMM_BLOCK_N;
  CUtensorMap ta;
  if (!MakeMapBf16(&ta, A, p.M, p.K, lda, a.a_box)) return -2;
  return LaunchPair<PAIR_W4>(ta, ta, p, a, min(DevicePairs(), a.n_pairs * a.m_tiles), stream);
}

// A: the experts' sorted token rows (fp16 or bf16 by `half`); the tile list of p.grp was built for tiles of `token_tile` rows (a multiple of 32)
int LaunchPairFp4(const void* A, int lda, const uint8_t* packed, const GemmParams& p, int token_tile, int max_tiles, bool half, cudaStream_t stream) {
  PairArgs a = {};
  a.n_pairs = (p.N + 255) / 256;
  a.bt = token_tile;
  a.a_box = token_tile / 2;
  a.packed = packed;
  a.n_tiles = (p.N + GEMM_BLOCK_N - 1) / GEMM_BLOCK_N;
  CUtensorMap ta;
  if (!MakeMapBf16(&ta, A, p.M, p.K, lda, a.a_box)) return -2;
  const int clusters = int(min((long long)DevicePairs(), (long long)a.n_pairs * max_tiles));
  return half ? LaunchPair<PAIR_FP4_F16>(ta, ta, p, a, clusters, stream) : LaunchPair<PAIR_FP4_BF16>(ta, ta, p, a, clusters, stream);
}

}  // namespace ogb
