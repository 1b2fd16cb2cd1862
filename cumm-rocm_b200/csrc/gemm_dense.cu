// gemm_dense.cu - dense GEMM of matmul2 (NoShuffle, 16-bit operands) on
// sm_100a tensor cores.
//
//   C[m, n] = act(alpha * op(A) @ op(B) + beta * D)
// with op(A) = A [m, k] or A^T (A stored [k, m]) and op(B) = B [k, n] or B^T
// (B stored [n, k]) -- the reference's GemmMainUnitTest.matmul2 without a
// shuffle (cumm/gemm/main.py:1176-1335, kernel cumm/gemm/kernel.py:586-940;
// split-K as in cumm/gemm/nvrtc_code.py:68-75 and params.h:115-132, here as a
// parallel reduction into an fp32 workspace instead of the serial semaphore).
//
// B200 design, two kernels: CTA pairs on 256 x 256 tiles where K is long
// (dense_gemm_pair_kernel; the rule is in launch_dense_gemm), and single CTAs
// on 128 x 256 tiles, or 128 x 128 and 128 x 64 with two CTAs per SM where K
// is short.  The single one, at 256 columns: persistent CTAs (one per SM) walk
// (128 x 256 output tile, K split) work units.  Warp 4 loads 128 x 64 A and 256 x 64 B blocks with
// 2-D TMA boxes into a 4-stage ring (48 KB per stage, SWIZZLE_128B); a
// row-major operand is K-major for the tensor core and a transposed one is
// read in place as MN-major (no copy).  Warp 5 issues tcgen05.mma (M = 128,
// N = 256, K = 16, 128 cycles each from one issuing thread: the tensor pipe's
// rate) into a double-buffered 128 x 256 fp32 TMEM
// accumulator, so warps 0-3 run the epilogue of one tile while the next one
// accumulates.  The epilogue applies act(alpha acc + beta D) and stores
// whole 128-byte lines, or with split-K adds its partial tile into an fp32
// workspace with red.global.add.v4.f32 (a finalize pass applies the
// epilogue).  Rows and columns past m / n / k are TMA zero fill on the loads
// and skipped on the stores.  Every mbarrier wait is bounded.
#include <cuda.h>

#include "kernels.h"

namespace scb {
namespace {

constexpr int kBM = 128, kBN = 256, kBK = 64;
constexpr int kMaxStages = 4;
constexpr int kThreads = 192;  // warps 0-3 epilogue, 4 TMA producer, 5 MMA issuer
constexpr int kWarpBuf = 4096;  // bytes per epilogue warp: 32 rows x 128 bytes
constexpr int kGroupM = 16;    // row tiles per raster group
constexpr uint32_t kABytes = kBM * kBK * 2;  // 16 KB

// CTA-pair kernel: a 256 x 256 tile per pair, 128 rows of A and 128 columns of
// B loaded by each CTA.  Six stages leave room for the epilogue's buffers; seven
// without them ran 8192^3 in 715 us against 686.
constexpr int kPairMinBlocks = 16;  // K blocks of a unit from which pairs are used
constexpr int kNarrowBlocks = 8;  // single CTAs: 128 columns up to this many K blocks
constexpr int kPairBM = 256;
constexpr int kPairStages = 6;
constexpr uint32_t kPairBBytes = kBN / 2 * kBK * 2;  // 16 KB
constexpr uint32_t kPairStageBytes = kABytes + kPairBBytes;

struct DParams {
  CUtensorMap ta;
  CUtensorMap tb;
  GemmArgs g;
  int a_mn, b_mn;  // operand is MN-major (stored transposed relative to the MMA's K-major form)
  int64_t m_tiles, n_tiles, units;
  int splits, kb_per_split, kblocks;
  int bn, stages;          // single-CTA kernel: columns of a tile, ring stages
  uint32_t stage_bytes;
  uint32_t bar_off;
  uint32_t idesc;
  float *ws;  // split-K: fp32 [m, n] (ld n), zeroed; else null
};

__device__ __forceinline__ void flag_error(int *err, int bits) { atomicOr(err, bits); }

// Output tile -> (row tile, column tile).  Tiles are walked in groups of
// kGroupM row tiles (half as many of the pair kernel's 256-row tiles), column by column inside a group, so the tiles that the
// persistent CTAs hold at one time (one each) cover a compact block: at
// 8192^3, 16 row tiles x ~10 column tiles = 34 MB of A and 42 MB of B, which
// stay in L2 instead of B streaming from HBM once per 4.6 row tiles.
template <int kGroup = kGroupM>
__device__ __forceinline__ void tile_mn(const DParams &P, int64_t tile, int64_t &mt, int64_t &nt) {
  const int64_t per_group = static_cast<int64_t>(kGroup) * P.n_tiles;
  const int64_t g = tile / per_group;
  const int64_t first = g * kGroup;
  const int64_t gm = P.m_tiles - first < kGroup ? P.m_tiles - first : kGroup;
  const int64_t r = tile - g * per_group;
  mt = first + r % gm;
  nt = r / gm;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void red_add_v4(float *p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

// act(alpha acc + beta D) of `ncol` (16: all) columns from col0 of output row `row`.
template <typename TOut>
__device__ __forceinline__ void apply16(const GemmArgs &G, int64_t row, int64_t col0, int64_t ncol, float *acc) {
  const EpiParams &e = G.epi;
  constexpr int kPer16 = 16 / sizeof(TOut);
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] *= e.alpha;
  if (e.beta != 0.f && e.src != nullptr) {
    const TOut *src = static_cast<const TOut *>(e.src) + row * e.src_ld + col0;
    if (ncol == 16 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
#pragma unroll
      for (int i = 0; i < 16; i += kPer16) {
        const uint4 q = *reinterpret_cast<const uint4 *>(src + i);
        const TOut *h = reinterpret_cast<const TOut *>(&q);
#pragma unroll
        for (int j = 0; j < kPer16; ++j) acc[i + j] = fmaf(e.beta, to_f32(h[j]), acc[i + j]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i < ncol) acc[i] = fmaf(e.beta, to_f32(src[i]), acc[i]);
      }
    }
  }
  apply_act_n<16>(acc, e.act_type, e.act_alpha);
}

// Epilogue of 16 accumulator columns [col0, col0 + 16) of output row `row`,
// stored (or, with split-K, added) by the row's own thread.
template <typename TOut>
__device__ __forceinline__ void store16(const DParams &P, int64_t row, int64_t col0, float *acc) {
  const GemmArgs &G = P.g;
  const int64_t ncol = G.n - col0 < 16 ? G.n - col0 : 16;
  if (P.ws != nullptr) {
    float *w = P.ws + row * G.n + col0;
    if (ncol == 16 && (G.n & 3) == 0) {
#pragma unroll
      for (int i = 0; i < 16; i += 4) red_add_v4(w + i, acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i < ncol) atomicAdd(w + i, acc[i]);
      }
    }
    return;
  }
  apply16<TOut>(G, row, col0, ncol, acc);
  TOut *dst = static_cast<TOut *>(G.c) + row * G.ldc + col0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (i < ncol) dst[i] = from_f32<TOut>(acc[i]);
  }
}

// Epilogue of one warp's 32 rows (from row0, TMEM address t0) x the tile's
// columns from nb.  Column blocks of 128 bytes go through the warp's 4 KB of
// shared memory (16-byte units XOR-swizzled by row) so that a store instruction
// writes four whole 128-byte lines; a row per thread wrote 32 pieces of 32
// lines (16384 x 4096 x 2048: 200 us, staged 187; 8192^3 762 / 750), and a
// block that n cuts went out in single elements (400000 x 32 x 32: 119 us,
// staged 36; 400000 x 96 x 256: 167 / 63).  Split-K, and rows that do not start
// or end on 16 bytes, are written by the rows' own threads.  With the
// activation's switch outside the element loop this took 8192 x 8192 x 256 from
// 367 to 138 us and 304 x 520 x 200 from 48 to 15: a tile's epilogue was longer
// than its mainloop up to K of about 4096.
template <typename TOut>
__device__ __forceinline__ void store_tile(const DParams &P, uint8_t *buf, int lane, int64_t row0, int64_t nb,
                                           uint32_t t0, bool any) {
  const GemmArgs &G = P.g;
  constexpr int kCols = 128 / sizeof(TOut);
  constexpr int kUnits = 16 * sizeof(TOut) / 16;  // 16-byte units of 16 columns
  const int64_t row = row0 + lane;
  const bool lines = P.ws == nullptr && (reinterpret_cast<uintptr_t>(G.c) & 15u) == 0 &&
                     (G.ldc * static_cast<int64_t>(sizeof(TOut))) % 16 == 0 && G.n % (16 / sizeof(TOut)) == 0;
  for (int cb = 0; cb < kBN; cb += kCols) {
    if (nb + cb >= G.n || cb >= P.bn) break;  // warp-uniform
    const int64_t left = G.n - nb - cb;  // columns from here
#pragma unroll
    for (int q = 0; q < kCols / 16; ++q) {
      const int64_t col0 = nb + cb + q * 16;
      if (col0 >= G.n) break;  // warp-uniform
      float acc[16];
      if (any) {
        tmem_ld16(t0 + static_cast<uint32_t>(cb + q * 16), acc);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
      }
      if (!lines) {
        if (row < G.m) store16<TOut>(P, row, col0, acc);
        continue;
      }
      if (row < G.m) apply16<TOut>(G, row, col0, left - q * 16 < 16 ? left - q * 16 : 16, acc);
#pragma unroll
      for (int u = 0; u < kUnits; ++u) {
        uint4 w;
        TOut *h = reinterpret_cast<TOut *>(&w);
#pragma unroll
        for (int j = 0; j < 16 / static_cast<int>(sizeof(TOut)); ++j)
          h[j] = from_f32<TOut>(acc[u * (16 / sizeof(TOut)) + j]);
        *reinterpret_cast<uint4 *>(buf + lane * 128 + (((q * kUnits + u) ^ (lane & 7)) << 4)) = w;
      }
    }
    if (!lines) continue;
    __syncwarp();
    const int unit = (lane & 7) * static_cast<int>(16 / sizeof(TOut));
    TOut *dst = static_cast<TOut *>(G.c) + nb + cb + unit;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + (lane >> 3);
      const uint4 w = *reinterpret_cast<const uint4 *>(buf + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
      if (row0 + r < G.m && unit < left) *reinterpret_cast<uint4 *>(dst + (row0 + r) * G.ldc) = w;
    }
    __syncwarp();
  }
}

template <typename TOut>
__global__ void __launch_bounds__(kThreads, 2) dense_gemm_kernel(const __grid_constant__ DParams P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u32 = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_u32 & 1023u)) & 1023u;
  uint8_t *smem = smem_raw + pad;
  const uint32_t smem_base = raw_u32 + pad;
  const GemmArgs &G = P.g;

  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + P.bar_off);
  uint64_t *full = bars;
  uint64_t *empty = bars + kMaxStages;
  uint64_t *acc_full = empty + kMaxStages;
  uint64_t *acc_empty = acc_full + 2;
  uint64_t *tile_bar = acc_empty + 2;
  uint64_t *drain_bar = tile_bar + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain_bar + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  volatile long long *acc_unit = reinterpret_cast<volatile long long *>(tmem_slot + 2);  // [2]
  volatile int *acc_nkb = reinterpret_cast<volatile int *>(tmem_slot + 6);              // [2]

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < P.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 128);
      mbar_init(&tile_bar[i], 1);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, 2 * P.bn);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 4) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      uint32_t stage = 0, eph = 0;
      bool ok = true;
      for (int64_t u = blockIdx.x; u < P.units && ok; u += gridDim.x) {
        const int64_t tile = u / P.splits;
        const int ks = static_cast<int>(u % P.splits);
        int64_t mt, nt;
        tile_mn(P, tile, mt, nt);
        const int m0 = static_cast<int>(mt * kBM);
        const int n0 = static_cast<int>(nt * P.bn);
        const int kb0 = ks * P.kb_per_split;
        const int kb1 = min(P.kblocks, kb0 + P.kb_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty[stage], eph ^ 1u, abort_flag)) {
            flag_error(G.err, kErrWaitTimeout);
            ok = false;
            break;
          }
          const uint32_t sA = smem_base + stage * P.stage_bytes;
          const uint32_t sB = sA + kABytes;
          const int k0 = kb * kBK;
          mbar_arrive_expect_tx(&full[stage], P.stage_bytes);
          if (P.a_mn) {
            tma_load_2d(sA, &P.ta, m0, k0, &full[stage]);
            tma_load_2d(sA + 8192, &P.ta, m0 + 64, k0, &full[stage]);
          } else {
            tma_load_2d(sA, &P.ta, k0, m0, &full[stage]);
          }
          if (P.b_mn) {
            for (int q = 0; q < P.bn / 64; ++q) tma_load_2d(sB + q * 8192, &P.tb, n0 + 64 * q, k0, &full[stage]);
          } else {
            tma_load_2d(sB, &P.tb, k0, n0, &full[stage]);
          }
          if (++stage == static_cast<uint32_t>(P.stages)) {
            stage = 0;
            eph ^= 1u;
          }
        }
      }
    }
  } else if (warp == 5) {
    // ---------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      uint32_t stage = 0, fph = 0;
      bool issued = false, ok = true;
      int it = 0;
      for (int64_t u = blockIdx.x;; u += gridDim.x, ++it) {
        const bool have = u < P.units;
        const int ab = it & 1;
        const uint32_t aph = (it >> 1) & 1;
        if (!mbar_wait(&acc_empty[ab], aph ^ 1u, abort_flag)) {
          flag_error(G.err, kErrWaitTimeout);
          break;
        }
        tc_fence_after();
        int nkb = 0;
        if (have) {
          const int ks = static_cast<int>(u % P.splits);
          const int kb0 = ks * P.kb_per_split;
          nkb = max(0, min(P.kblocks, kb0 + P.kb_per_split) - kb0);
        }
        acc_unit[ab] = have ? u : -1;
        acc_nkb[ab] = nkb;
        mbar_arrive(&tile_bar[ab]);
        if (!have) break;
        const uint32_t d = tmem_base + static_cast<uint32_t>(ab * P.bn);
        for (int j = 0; j < nkb; ++j) {
          if (!mbar_wait(&full[stage], fph, abort_flag)) {
            flag_error(G.err, kErrWaitTimeout);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sA = smem_base + stage * P.stage_bytes;
          const uint32_t sB = sA + kABytes;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            // K advances 16 elements: 32 bytes inside a K-major row, 16 rows
            // (2 KB) of an MN-major atom
            const uint64_t ad = P.a_mn ? make_sdesc(sA + kk * 2048, 8192, 1024) : make_sdesc(sA + kk * 32, 16, 1024);
            const uint64_t bd = P.b_mn ? make_sdesc(sB + kk * 2048, 8192, 1024) : make_sdesc(sB + kk * 32, 16, 1024);
            mma_f16(d, ad, bd, P.idesc, (j | kk) != 0 ? 1u : 0u);
          }
          issued = true;
          mma_commit(&empty[stage]);
          if (++stage == static_cast<uint32_t>(P.stages)) {
            stage = 0;
            fph ^= 1u;
          }
        }
        if (!ok) break;
        if (nkb == 0) mbar_arrive(&acc_full[ab]);
        else mma_commit(&acc_full[ab]);
      }
      if (issued) {
        mma_commit(drain_bar);
        int never = 0;
        if (!mbar_wait(drain_bar, 0, reinterpret_cast<volatile int *>(&never))) flag_error(G.err, kErrWaitTimeout);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 0-3)
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    for (int it = 0;; ++it) {
      const int ab = it & 1;
      const uint32_t aph = (it >> 1) & 1;
      if (!mbar_wait(&tile_bar[ab], aph, abort_flag)) {
        flag_error(G.err, kErrWaitTimeout);
        break;
      }
      const long long u = acc_unit[ab];
      if (u < 0) break;
      const int nkb = acc_nkb[ab];
      if (!mbar_wait(&acc_full[ab], aph, abort_flag)) {
        flag_error(G.err, kErrWaitTimeout);
        break;
      }
      tc_fence_after();
      const int64_t tile = u / P.splits;
      int64_t mt, nt;
      tile_mn(P, tile, mt, nt);
      store_tile<TOut>(P, smem + P.stages * P.stage_bytes + warp * kWarpBuf, lane, mt * kBM + warp * 32, nt * P.bn,
                       tmem_base + lane_base + static_cast<uint32_t>(ab * P.bn), nkb > 0);
      tc_fence_before();
      mbar_arrive(&acc_empty[ab]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * P.bn);
  }
}

// ---- CTA pair (cta_group::2) primitives
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Shared-window address of `addr` in the pair's leader (rank 0).
__device__ __forceinline__ uint32_t leader_smem(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void mbar_arrive_leader(uint32_t leader_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_bar) : "memory");
}
// 2-D box into this CTA's shared memory; the bytes complete on the leader's barrier.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y,
                                                 uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once the pair's MMAs so far are done.
__device__ __forceinline__ void mma_commit_pair(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

// One 256 x 256 tile per CTA pair (cta_group::2): the tensor core reads both
// CTAs' B halves, so a CTA stages 32 KB per 64 K-elements instead of 48, moves
// a third less through L2 and holds six stages instead of four; a pair's MMA
// (M = 256, N = 256, K = 16) takes the 128 cycles of the single one's
// M = 128.  Rank 0's MMA warp issues for both; its full barriers count both
// CTAs' loads, and its commits release the stages of both.  The sums are the
// single kernel's, in its order.  8192^3 alone: 750 -> 686 us; after other work,
// with L2 flushed, 724 (1,519 TFLOP/s; cuBLAS 679 in the same run).  What is left is the tensor pipe at the clock that the power limit allows, and the
// last wave (1,024 units on 74 pairs: 13.8 waves).
template <typename TOut>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    dense_gemm_pair_kernel(const __grid_constant__ DParams P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_u32 = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_u32 & 1023u)) & 1023u;  // the same in both CTAs
  uint8_t *smem = smem_raw + pad;
  const uint32_t smem_base = raw_u32 + pad;
  const GemmArgs &G = P.g;

  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + P.bar_off);
  uint64_t *full = bars;                    // leader's: both CTAs' loads
  uint64_t *empty = full + kPairStages;     // each CTA's: the pair's MMAs have read the stage
  uint64_t *acc_full = empty + kPairStages; // each CTA's
  uint64_t *acc_empty = acc_full + 2;       // leader's: both CTAs' epilogue threads
  uint64_t *drain_bar = acc_empty + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain_bar + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int64_t first = blockIdx.x >> 1;
  const int64_t step = gridDim.x >> 1;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPairStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 256);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 4) {
    // ---------------------------------------------------------------- TMA producer (both CTAs)
    if (elect_one()) {
      uint32_t stage = 0, eph = 0;
      bool ok = true;
      for (int64_t u = first; u < P.units && ok; u += step) {
        const int64_t tile = u / P.splits;
        const int ks = static_cast<int>(u % P.splits);
        int64_t mt, nt;
        tile_mn<kGroupM / 2>(P, tile, mt, nt);
        const int m0 = static_cast<int>(mt * kPairBM) + static_cast<int>(rank) * kBM;
        const int n0 = static_cast<int>(nt * kBN) + static_cast<int>(rank) * (kBN / 2);
        const int kb0 = ks * P.kb_per_split;
        const int kb1 = min(P.kblocks, kb0 + P.kb_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty[stage], eph ^ 1u, abort_flag)) {
            flag_error(G.err, kErrWaitTimeout);
            ok = false;
            break;
          }
          const uint32_t sA = smem_base + stage * kPairStageBytes;
          const uint32_t sB = sA + kABytes;
          const int k0 = kb * kBK;
          // A peer's bytes may land before the leader expects them: the phase
          // cannot end before the leader's one arrival.
          if (rank == 0) mbar_arrive_expect_tx(&full[stage], 2 * kPairStageBytes);
          const uint32_t bar = leader_smem(smem_u32(&full[stage]));
          if (P.a_mn) {
            tma_load_2d_pair(sA, &P.ta, m0, k0, bar);
            tma_load_2d_pair(sA + 8192, &P.ta, m0 + 64, k0, bar);
          } else {
            tma_load_2d_pair(sA, &P.ta, k0, m0, bar);
          }
          if (P.b_mn) {
            tma_load_2d_pair(sB, &P.tb, n0, k0, bar);
            tma_load_2d_pair(sB + 8192, &P.tb, n0 + 64, k0, bar);
          } else {
            tma_load_2d_pair(sB, &P.tb, k0, n0, bar);
          }
          if (++stage == kPairStages) {
            stage = 0;
            eph ^= 1u;
          }
        }
      }
    }
  } else if (warp == 5) {
    // ---------------------------------------------------------------- MMA issuer (leader only)
    if (rank == 0 && elect_one()) {
      uint32_t stage = 0, fph = 0;
      bool ok = true;
      int it = 0;
      for (int64_t u = first; u < P.units && ok; u += step, ++it) {
        const int ab = it & 1;
        const uint32_t aph = (it >> 1) & 1;
        if (!mbar_wait(&acc_empty[ab], aph ^ 1u, abort_flag)) {
          flag_error(G.err, kErrWaitTimeout);
          break;
        }
        tc_fence_after();
        const int kb0 = static_cast<int>(u % P.splits) * P.kb_per_split;
        const int nkb = max(0, min(P.kblocks, kb0 + P.kb_per_split) - kb0);
        const uint32_t d = tmem_base + static_cast<uint32_t>(ab * kBN);
        for (int j = 0; j < nkb; ++j) {
          if (!mbar_wait(&full[stage], fph, abort_flag)) {
            flag_error(G.err, kErrWaitTimeout);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sA = smem_base + stage * kPairStageBytes;
          const uint32_t sB = sA + kABytes;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint64_t ad = P.a_mn ? make_sdesc(sA + kk * 2048, 8192, 1024) : make_sdesc(sA + kk * 32, 16, 1024);
            const uint64_t bd = P.b_mn ? make_sdesc(sB + kk * 2048, 8192, 1024) : make_sdesc(sB + kk * 32, 16, 1024);
            mma_f16_pair(d, ad, bd, P.idesc, (j | kk) != 0 ? 1u : 0u);
          }
          mma_commit_pair(&empty[stage]);
          if (++stage == kPairStages) {
            stage = 0;
            fph ^= 1u;
          }
        }
        if (ok) mma_commit_pair(&acc_full[ab]);
      }
      mma_commit_pair(drain_bar);
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- epilogue (warps 0-3, both CTAs)
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    int it = 0;
    for (int64_t u = first; u < P.units; u += step, ++it) {
      const int ab = it & 1;
      const uint32_t aph = (it >> 1) & 1;
      const int64_t tile = u / P.splits;
      const int kb0 = static_cast<int>(u % P.splits) * P.kb_per_split;
      const bool any = kb0 < P.kblocks;
      if (!mbar_wait(&acc_full[ab], aph, abort_flag)) {
        flag_error(G.err, kErrWaitTimeout);
        break;
      }
      tc_fence_after();
      int64_t mt, nt;
      tile_mn<kGroupM / 2>(P, tile, mt, nt);
      store_tile<TOut>(P, smem + kPairStages * kPairStageBytes + warp * kWarpBuf, lane,
                       mt * kPairBM + static_cast<int64_t>(rank) * kBM + warp * 32, nt * kBN,
                       tmem_base + lane_base + static_cast<uint32_t>(ab * kBN), any);
      tc_fence_before();
      mbar_arrive_leader(leader_smem(smem_u32(&acc_empty[ab])));
    }
  }

  // Neither CTA leaves while the pair's MMAs may still read its shared memory,
  // write its TMEM or signal its barriers; every wait is bounded, so both come here.
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) {
    int never = 0;
    if (!mbar_wait(drain_bar, 0, reinterpret_cast<volatile int *>(&never))) flag_error(G.err, kErrWaitTimeout);
  }
  __syncthreads();
  cluster_sync_all();
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
  }
}

}  // namespace

bool dense_gemm_supported(const GemmArgs &a) {
  if (a.shuffle != 0) return false;
  if (a.in_dtype != 12 && a.in_dtype != 7) return false;
  if (a.out_dtype != 0 && a.out_dtype != 7 && a.out_dtype != 12) return false;
  if ((a.lda * 2) % 16 || (a.ldb * 2) % 16) return false;
  if (reinterpret_cast<uintptr_t>(a.a) % 16 || reinterpret_cast<uintptr_t>(a.b) % 16) return false;
  if (a.m <= 0 || a.n <= 0 || a.k < 0) return false;
  return true;
}

int dense_gemm_splits(const GemmArgs &a) {
  const int64_t kblocks = (a.k + kBK - 1) / kBK;
  int s = a.split_k > 1 ? a.split_k : 1;
  if (s > kblocks) s = static_cast<int>(kblocks > 0 ? kblocks : 1);
  return s;
}

cudaError_t launch_dense_gemm(const GemmArgs &a, float *split_ws, int num_sms, cudaStream_t stream) {
  DParams P;
  P.g = a;
  const int splits = dense_gemm_splits(a);
  P.kblocks = static_cast<int>((a.k + kBK - 1) / kBK);
  P.splits = splits;
  P.kb_per_split = P.kblocks > 0 ? (P.kblocks + P.splits - 1) / P.splits : 0;
  // A short K leaves a tile to its epilogue, so it gets narrow tiles: room for
  // two CTAs (and epilogues) per SM, and no loads for the padding columns of a
  // narrow output (1x1x1 convolutions over voxels).  us, 256 columns / narrow:
  // 400000 x 64 x 64 54 / 35 (64 columns), 400000 x 128 x 128 81 / 54 (128),
  // 200000 x 64 x 512 84 / 52; outputs wider than the tile (128): 400000 x 256
  // x 256 136 / 105, 8192 x 8192 x 256 90 / 72, x 512 98 / 86, x 960 111 / 139
  // (the ring of two stages).  With K of 2048 even 128 columns took 174 us in
  // narrow tiles against 160 in pairs, so a long K keeps 256.
  const bool narrow = P.kb_per_split < kPairMinBlocks;
  P.bn = narrow && a.n <= 64 ? 64 : (narrow && a.n <= 128) || P.kb_per_split <= kNarrowBlocks ? 128 : kBN;
  const int64_t n_tiles = (a.n + P.bn - 1) / P.bn;
  const int64_t units1 = (a.m + kBM - 1) / kBM * n_tiles * splits;
  const int64_t units2 = (a.m + kPairBM - 1) / kPairBM * n_tiles * splits;
  // A second CTA per SM only where there are tiles for it; else the whole ring.
  const bool two = P.bn < kBN && units1 > num_sms;
  P.stages = !two ? kMaxStages : P.bn == 64 ? 3 : 2;
  P.stage_bytes = kABytes + static_cast<uint32_t>(P.bn) * kBK * 2;
  // CTA pairs where the mainloop is long enough to bound a tile: K >= 1024 per
  // unit.  us, single / pair: 8192 x 8192 x K with K = 512: 90 / 96, 1024:
  // 104 / 104, 1536: 144 / 125, 2048: 188 / 158; 60000 x 512 x K: 51 / 53,
  // 66 / 64, 86 / 76, 107 / 92; 256 x 8192 x K: 16 / 18, 21 / 21, 25 / 23,
  // 27 / 25.  Below that the epilogue bounds the tile.  And only where 256-row tiles take no more
  // waves: 1152 x 8192 x 4096 is 288 units in 2 waves of 148, or 160 in 3 waves
  // of 74 (68 / 76); 1280 rows take 3 either way (95 / 79).
  const int pairs = num_sms / 2;
  const bool pair = P.bn == kBN && P.kb_per_split >= kPairMinBlocks && pairs > 0 &&
                    (units2 + pairs - 1) / pairs <= (units1 + num_sms - 1) / num_sms;
  P.a_mn = a.trans_a ? 1 : 0;
  P.b_mn = a.trans_b ? 0 : 1;
  // A: [m, k] (K-major, 64 x 128 boxes) or stored [k, m] (MN-major, 64 x 64 boxes)
  const bool ok_a = P.a_mn ? encode_tmap_2d(&P.ta, a.in_dtype, a.a, static_cast<uint64_t>(a.m),
                                            static_cast<uint64_t>(a.k > 0 ? a.k : 1),
                                            static_cast<uint64_t>(a.lda) * 2, 64, 64)
                           : encode_tmap_2d(&P.ta, a.in_dtype, a.a, static_cast<uint64_t>(a.k > 0 ? a.k : 1),
                                            static_cast<uint64_t>(a.m), static_cast<uint64_t>(a.lda) * 2, 64, kBM);
  // B: stored [n, k] (K-major, 64 x 256 boxes) or [k, n] (MN-major, 64 x 64 boxes)
  const bool ok_b = P.b_mn ? encode_tmap_2d(&P.tb, a.in_dtype, a.b, static_cast<uint64_t>(a.n),
                                            static_cast<uint64_t>(a.k > 0 ? a.k : 1),
                                            static_cast<uint64_t>(a.ldb) * 2, 64, 64)
                           : encode_tmap_2d(&P.tb, a.in_dtype, a.b, static_cast<uint64_t>(a.k > 0 ? a.k : 1),
                                            static_cast<uint64_t>(a.n), static_cast<uint64_t>(a.ldb) * 2, 64, pair ? kBN / 2 : P.bn);
  if (!ok_a || !ok_b) return cudaErrorInvalidValue;
  P.m_tiles = pair ? (a.m + kPairBM - 1) / kPairBM : (a.m + kBM - 1) / kBM;
  P.n_tiles = n_tiles;
  P.units = pair ? units2 : units1;
  P.ws = P.splits > 1 ? split_ws : nullptr;
  P.bar_off = (pair ? kPairStages * kPairStageBytes : P.stages * P.stage_bytes) + 4 * kWarpBuf;
  P.idesc = make_idesc(pair ? kPairBM : kBM, P.bn, a.in_dtype == 12 ? 1u : 0u, P.a_mn != 0, P.b_mn != 0);
  const size_t smem = 1024 + P.bar_off + 256;
  const int64_t ctas = two ? 2 * num_sms : num_sms;
  const int grid = pair ? 2 * static_cast<int>(units2 < pairs ? units2 : pairs)
                        : static_cast<int>(units1 < ctas ? units1 : ctas);
  void (*kern)(DParams);
  switch (a.out_dtype) {
    case 0: kern = pair ? dense_gemm_pair_kernel<float> : dense_gemm_kernel<float>; break;
    case 7: kern = pair ? dense_gemm_pair_kernel<__half> : dense_gemm_kernel<__half>; break;
    case 12: kern = pair ? dense_gemm_pair_kernel<__nv_bfloat16> : dense_gemm_kernel<__nv_bfloat16>; break;
    default: return cudaErrorInvalidValue;
  }
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  kern<<<grid, kThreads, smem, stream>>>(P);
  return cudaGetLastError();
}

}  // namespace scb
