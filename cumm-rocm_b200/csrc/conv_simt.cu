// conv_simt.cu - fp32 mask-implicit-GEMM sparse convolution with FFMA.
//
// The fp32 path (reference algo "Simt", cumm/gemm/algospec/simt.py) keeps full
// fp32 products so results stay within 1e-5 of an fp64 evaluation; tensor-core
// tf32 would not.  Semantics are those of the tcgen05 kernels:
//   fwd / dgrad: the tile mask (OR of the masks of tile_shape[0] sorted rows AND
//     mask_filter, reversed for dgrad with reverse_mask) selects the offsets
//     (cumm/conv/kernel.py:844-889); row r gathers A[indices[k][sigma(r)]] and
//     the result goes to row sigma(r).
//   wgrad: dW[:, k, :] += dOut[sigma(r)]^T In[indices[k][sigma(r)]] over rows r
//     whose reduced mask word mask[r / mask_width] has bit k
//     (cumm/gemm/blockmma/mma.py:580-765), accumulated into an fp32 workspace.
//
// Both kernels read a block's indices once (two round trips for all offsets or
// rows), then run a three-stage cp.async ring over 32-element slices, so the
// gathers of the next slices are in flight while one is multiplied.  Rows move
// in 16-byte copies when row lengths and base pointers allow it, else in
// 4-byte ones.  Bound: shared-memory reads of the register tiles, and blocks
// per SM at small clouds.  20k voxels, C = K = 32, against one block per
// 128-row tile with an index load, a row load and a barrier per slice: forward
// 453 -> 59 us, backward-input 449 -> 58, backward-weight 433 -> 42.
// A 16 x 1 register tile (one address per warp and A read) was slower: 67 us.
#include "kernels.h"
#include "launch_rules.h"

namespace scb {
namespace {

constexpr int kSlice = 32;           // reduction elements per stage
constexpr int kPitch = kSlice + 4;   // floats between rows of a [row][slice] tile: 16-byte aligned, conflict-free
constexpr int kStages = 3;
constexpr int kMaxGridYZ = 65535;    // more blocks along y or z take several launches

__device__ __forceinline__ uint32_t smem_addr(const float *p) { return smem_u32(p); }

// `count` floats (<= 4) of a 16-byte unit; absent ones become zeros.
template <bool kVec>
__device__ __forceinline__ void copy4(float *dst, const float *src, const float *any, int count) {
  if constexpr (kVec) {
    cp_async_16(smem_addr(dst), count > 0 ? src : any, count > 0 ? 16u : 0u);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) cp_async_4(smem_addr(dst + q), q < count ? src + q : any, q < count ? 4u : 0u);
  }
}

// One block: kRows sorted rows x kCols output columns, kRows / 4 x 8 threads,
// each 4 rows x kCols / 8 columns.  Sums run over the offsets, then the
// reduction elements, in ascending order.
template <bool kFwd, bool kVec, int kRows, int kCols>
__global__ void __launch_bounds__(kRows * 2)
simt_fwd_kernel(const ConvSimtArgs A, int n_red, int n_out, int col_block0) {
  constexpr int kThreads = kRows * 2;
  constexpr int kPer = kCols / 8;
  constexpr int kATile = kRows * kPitch;
  constexpr int kBPitch = kCols + 4;                                   // dgrad: B as [slice][column]
  constexpr int kBTile = kFwd ? kCols * kPitch : kSlice * kBPitch;     // fwd: B as [column][slice]
  extern __shared__ __align__(16) float sm[];
  float *ring = sm;
  int *s_idx = reinterpret_cast<int *>(sm + kStages * (kATile + kBTile));  // [slot][kRows]
  __shared__ uint32_t s_km;
  __shared__ int s_sig[kRows];
  __shared__ int s_k[32];
  const int tid = threadIdx.x;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * kRows;
  const int nb = (col_block0 + static_cast<int>(blockIdx.y)) * kCols;
  if (tid == 0) s_km = 0;
  __syncthreads();
  // the mask tile may be wider than the block's rows
  const int64_t mask0 = row0 / A.tile_m_desp * A.tile_m_desp;
  uint32_t m = 0;
  for (int r = tid; r < A.tile_m_desp; r += kThreads)
    if (mask0 + r < A.M) m |= A.mask[mask0 + r];
  if (m) atomicOr(&s_km, m);
  if (tid < kRows) {
    int sig = -1;
    if (row0 + tid < A.M) {
      sig = A.argsort[row0 + tid];
      if (sig < 0 || sig >= A.M) {
        atomicOr(A.err, kErrBadIndex);
        sig = -1;
      }
    }
    s_sig[tid] = sig;
  }
  __syncthreads();
  uint32_t km = s_km & A.mask_filter;
  if (kFwd && A.mask_out != nullptr && tid == 0 && nb == 0 && row0 == mask0)
    A.mask_out[row0 / A.tile_m_desp] = km;
  if (!kFwd && km == 0) return;  // dgrad early exit (kernel.py:875-882)
  if (!kFwd && A.reverse) km = __brev(km) >> (32 - A.kv);
  const int n_off = __popc(km);
  if (tid < 32 && ((km >> tid) & 1u)) s_k[__popc(km & ((1u << tid) - 1u))] = tid;
  __syncthreads();
  for (int e = tid; e < n_off * kRows; e += kThreads) {
    const int sg = s_sig[e % kRows];
    int idx = -1;
    if (sg >= 0) {
      idx = A.indices[static_cast<int64_t>(s_k[e / kRows]) * A.M + sg];
      if (idx < -1 || idx >= A.a_rows) {
        atomicOr(A.err, kErrBadIndex);
        idx = -1;
      }
    }
    s_idx[e] = idx;
  }
  __syncthreads();

  const int slices = (n_red + kSlice - 1) / kSlice;
  const int chunks = n_off * slices;
  int l_slot = 0, l_c0 = 0;  // chunk to load next
  auto load = [&](int stage) {
    float *sA = ring + stage * (kATile + kBTile);
    float *sB = sA + kATile;
    const int k = s_k[l_slot];
    const int *idx = s_idx + l_slot * kRows;
    for (int e = tid; e < kRows * (kSlice / 4); e += kThreads) {
      const int r = e / (kSlice / 4), u = (e % (kSlice / 4)) * 4;
      const int i = idx[r];
      const int left = i >= 0 ? n_red - l_c0 - u : 0;
      copy4<kVec>(sA + r * kPitch + u, A.a + static_cast<int64_t>(i < 0 ? 0 : i) * n_red + l_c0 + u, A.a, left);
    }
    if constexpr (kFwd) {  // W[n, k, c]
      for (int e = tid; e < kCols * (kSlice / 4); e += kThreads) {
        const int n = e / (kSlice / 4), u = (e % (kSlice / 4)) * 4;
        const int left = nb + n < n_out ? n_red - l_c0 - u : 0;
        copy4<kVec>(sB + n * kPitch + u, A.b + (static_cast<int64_t>(nb + n) * A.kv + k) * n_red + l_c0 + u, A.b, left);
      }
    } else {               // W[c_red, k, n], n = input channel
      for (int e = tid; e < kSlice * (kCols / 4); e += kThreads) {
        const int c = e / (kCols / 4), u = (e % (kCols / 4)) * 4;
        const int left = l_c0 + c < n_red ? n_out - nb - u : 0;
        copy4<kVec>(sB + c * kBPitch + u, A.b + (static_cast<int64_t>(l_c0 + c) * A.kv + k) * n_out + nb + u, A.b, left);
      }
    }
    l_c0 += kSlice;
    if (l_c0 >= n_red) {
      l_c0 = 0;
      ++l_slot;
    }
  };

  const int cg = tid & 7;   // fwd: columns cg + 8 j; dgrad: 4 cg + (j & 3) + 32 (j >> 2)
  const int rg = tid >> 3;  // rows rg + kRows / 4 * i
  float acc[4][kPer];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < kPer; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int q = 0; q < kStages - 1; ++q) {
    if (q < chunks) load(q);
    cp_async_commit();
  }
  for (int ch = 0; ch < chunks; ++ch) {
    cp_async_wait<kStages - 2>();
    __syncthreads();  // chunk ch has landed; every thread is past chunk ch - 1
    if (ch + kStages - 1 < chunks) load((ch + kStages - 1) % kStages);
    cp_async_commit();
    const float *sA = ring + (ch % kStages) * (kATile + kBTile);
    const float *sB = sA + kATile;
#pragma unroll 2
    for (int c = 0; c < kSlice; c += 4) {
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4 *>(sA + (rg + kRows / 4 * i) * kPitch + c);
      float b[4][kPer];  // [element][column]
      if constexpr (kFwd) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          const float4 v = *reinterpret_cast<const float4 *>(sB + (cg + 8 * j) * kPitch + c);
          b[0][j] = v.x;
          b[1][j] = v.y;
          b[2][j] = v.z;
          b[3][j] = v.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int j = 0; j < kPer; j += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(sB + (c + q) * kBPitch + 4 * cg + 8 * j);
            b[q][j] = v.x;
            b[q][j + 1] = v.y;
            b[q][j + 2] = v.z;
            b[q][j + 3] = v.w;
          }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          acc[i][j] = fmaf(a[i].x, b[0][j], acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b[1][j], acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[2][j], acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b[3][j], acc[i][j]);
        }
    }
  }

  const EpiParams &e = A.epi;
  const float *src = static_cast<const float *>(e.src);
  const bool use_src = e.beta != 0.f && src != nullptr;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int sg = s_sig[rg + kRows / 4 * i];
    if (sg < 0) continue;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int n = nb + (kFwd ? cg + 8 * j : 4 * cg + (j & 3) + 32 * (j >> 2));
      if (n >= n_out) continue;
      float v;
      if (e.mode == 1) {
        const float sc = e.scale ? e.scale[n] : 1.f;
        v = sc * acc[i][j] + (e.bias ? e.alpha * static_cast<const float *>(e.bias)[n] : 0.f);
      } else {
        v = e.alpha * acc[i][j];
      }
      if (use_src) v = fmaf(e.beta, src[static_cast<int64_t>(sg) * e.src_ld + n], v);
      A.out[static_cast<int64_t>(sg) * n_out + n] = apply_act(v, e.act_type, e.act_alpha);
    }
  }
}

// dW tile of 32 x 32 (n, c) of one offset over one range of rows; grid: (kv,
// ceil(K / 32) * ceil(C / 32), row ranges).  The four warps take a quarter of
// each 64-row chunk's rows and every one holds the whole tile (4 n x 8 c per
// thread); their partial tiles are added with v4 reductions.
constexpr int kWThreads = 128;
constexpr int kWChunk = 64;          // rows per stage
constexpr int kWRange = 1024;        // most rows per block: 16 chunks, a bit each in s_some

template <bool kVec>
__global__ void __launch_bounds__(kWThreads)
simt_wgrad_kernel(const ConvSimtArgs A, int rows_per_block, int vec_out, int64_t row_block0) {
  extern __shared__ __align__(16) float sm[];  // [kStages][2][kWChunk][32]
  __shared__ int s_sig[kWRange], s_idx[kWRange];
  __shared__ unsigned s_some;
  const int k = blockIdx.x;
  const int ncb = (A.C + 31) / 32;
  const int n0 = (blockIdx.y / ncb) * 32;
  const int c0 = (blockIdx.y % ncb) * 32;
  const int64_t r0 = (row_block0 + blockIdx.z) * rows_per_block;
  const int rows = static_cast<int>(min(static_cast<int64_t>(rows_per_block), A.M - r0));
  const int tid = threadIdx.x;
  if (!((A.mask_filter >> k) & 1u)) return;
  if (tid == 0) s_some = 0u;
  __syncthreads();
  // rows and their inputs; a row whose mask word lacks the offset has none
  unsigned mine = 0u;
  for (int r = tid; r < rows; r += kWThreads) {
    const int64_t row = r0 + r;
    const int64_t wi = row / A.mask_width;
    const uint32_t word = wi < A.mask_count ? A.mask[wi] : 0u;
    int sg = A.argsort[row], idx = -1;
    if (sg < 0 || sg >= A.M) {
      atomicOr(A.err, kErrBadIndex);
      sg = -1;
    } else if ((word >> k) & 1u) {
      idx = A.indices[static_cast<int64_t>(k) * A.M + sg];
      if (idx < -1 || idx >= A.b_rows) {
        atomicOr(A.err, kErrBadIndex);
        idx = -1;
      }
    }
    s_sig[r] = sg;
    s_idx[r] = idx;
    if ((word >> k) & 1u) mine |= 1u << (r / kWChunk);
  }
  if (mine) atomicOr(&s_some, mine);
  __syncthreads();
  // chunks with a selected row
  const unsigned some = s_some;
  const int chunks = __popc(some);
  if (chunks == 0) return;

  unsigned to_load = some;  // loads go in order
  auto load = [&](int stage) {
    float *sO = sm + stage * 2 * kWChunk * 32;
    float *sI = sO + kWChunk * 32;
    const int base = (__ffs(to_load) - 1) * kWChunk;
    to_load &= to_load - 1u;
    for (int e = tid; e < kWChunk * 8; e += kWThreads) {
      const int r = base + e / 8, u = (e % 8) * 4;
      const int sg = r < rows ? s_sig[r] : -1;
      const int idx = r < rows ? s_idx[r] : -1;
      copy4<kVec>(sO + e * 4, A.a + static_cast<int64_t>(sg < 0 ? 0 : sg) * A.K + n0 + u, A.a, sg >= 0 ? A.K - n0 - u : 0);
      copy4<kVec>(sI + e * 4, A.b + static_cast<int64_t>(idx < 0 ? 0 : idx) * A.C + c0 + u, A.b,
                  idx >= 0 ? A.C - c0 - u : 0);
    }
  };
  const int lane = tid & 31, w = tid >> 5;
  const int tn = (lane >> 2) * 4, tc = (lane & 3) * 4;  // n: tn + i; c: tc + 16 (j / 4) + j % 4
  float acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int q = 0; q < kStages - 1; ++q) {
    if (q < chunks) load(q);
    cp_async_commit();
  }
  for (int ch = 0; ch < chunks; ++ch) {
    cp_async_wait<kStages - 2>();
    __syncthreads();
    if (ch + kStages - 1 < chunks) load((ch + kStages - 1) % kStages);
    cp_async_commit();
    const float *sO = sm + (ch % kStages) * 2 * kWChunk * 32 + w * (kWChunk / 4) * 32;
    const float *sI = sO + kWChunk * 32;
#pragma unroll 4
    for (int r = 0; r < kWChunk / 4; ++r) {
      const float4 o = *reinterpret_cast<const float4 *>(sO + r * 32 + tn);
      const float4 x = *reinterpret_cast<const float4 *>(sI + r * 32 + tc);
      const float4 y = *reinterpret_cast<const float4 *>(sI + r * 32 + tc + 16);
      const float on[4] = {o.x, o.y, o.z, o.w};
      const float in[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(on[i], in[j], acc[i][j]);
    }
  }
  // add the four warps' tiles in shared memory, then one reduction per block
  cp_async_wait_all();
  __syncthreads();
  float *part = sm + w * 32 * 32;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; j += 4)
      *reinterpret_cast<float4 *>(part + (tn + i) * 32 + tc + 4 * j) =
          make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
  __syncthreads();
  for (int e = tid; e < 32 * 8; e += kWThreads) {
    const int n = n0 + e / 8, c = c0 + (e % 8) * 4;
    float4 v = *reinterpret_cast<const float4 *>(sm + e * 4);
#pragma unroll
    for (int q = 1; q < 4; ++q) {
      const float4 p = *reinterpret_cast<const float4 *>(sm + q * 1024 + e * 4);
      v.x += p.x;
      v.y += p.y;
      v.z += p.z;
      v.w += p.w;
    }
    if (n >= A.K || c >= A.C) continue;
    float *dst = A.out + (static_cast<int64_t>(n) * A.kv + k) * A.C + c;
    if (vec_out) {
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                   : "memory");
    } else {
      const float f[4] = {v.x, v.y, v.z, v.w};
      for (int q = 0; q < 4 && c + q < A.C; ++q) atomicAdd(dst + q, f[q]);
    }
  }
}

bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

template <bool kFwd, bool kVec, int kRows, int kCols>
cudaError_t launch_fwd(const ConvSimtArgs &a, int n_red, int n_out, cudaStream_t stream) {
  constexpr int b_tile = kFwd ? kCols * kPitch : kSlice * (kCols + 4);
  const int smem = (kStages * (kRows * kPitch + b_tile) + 32 * kRows) * static_cast<int>(sizeof(float));
  auto kern = simt_fwd_kernel<kFwd, kVec, kRows, kCols>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int cols = (n_out - 1) / kCols + 1;
  for (int c0 = 0; c0 < cols; c0 += kMaxGridYZ) {
    const dim3 grid(static_cast<unsigned>((a.M + kRows - 1) / kRows), cols - c0 < kMaxGridYZ ? cols - c0 : kMaxGridYZ);
    kern<<<grid, kRows * 2, smem, stream>>>(a, n_red, n_out, c0);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <bool kFwd, bool kVec>
cudaError_t pick_fwd(const ConvSimtArgs &a, int n_red, int n_out, int num_sms, cudaStream_t stream) {
  // 64 rows a block where the mask tile has them; 64 columns (half the reads
  // of A per product) where they exist and the rows alone fill the GPU
  const bool wide = simt_wide_columns(a.M, n_out, num_sms);
  if (a.tile_m_desp == 32)
    return wide ? launch_fwd<kFwd, kVec, 32, 64>(a, n_red, n_out, stream)
                : launch_fwd<kFwd, kVec, 32, 32>(a, n_red, n_out, stream);
  return wide ? launch_fwd<kFwd, kVec, 64, 64>(a, n_red, n_out, stream)
              : launch_fwd<kFwd, kVec, 64, 32>(a, n_red, n_out, stream);
}

}  // namespace

cudaError_t launch_conv_simt(const ConvSimtArgs &a, int num_sms, cudaStream_t stream) {
  if (a.M == 0) return cudaSuccess;
  const bool vec = aligned16(a.a) && aligned16(a.b);
  if (a.op == 2) {
    const int64_t rows = simt_wgrad_rows(a.M, a.kv * ((a.K + 31) / 32) * ((a.C + 31) / 32), num_sms, kWChunk, kWRange);
    const bool v = vec && a.K % 4 == 0 && a.C % 4 == 0;
    const int vec_out = a.C % 4 == 0 && aligned16(a.out);
    auto kern = v ? simt_wgrad_kernel<true> : simt_wgrad_kernel<false>;
    const int smem = kStages * 2 * kWChunk * 32 * static_cast<int>(sizeof(float));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int64_t blocks = (a.M + rows - 1) / rows;
    for (int64_t z0 = 0; z0 < blocks; z0 += kMaxGridYZ) {
      const dim3 grid(a.kv, ((a.K + 31) / 32) * ((a.C + 31) / 32),
                      static_cast<unsigned>(blocks - z0 < kMaxGridYZ ? blocks - z0 : kMaxGridYZ));
      kern<<<grid, kWThreads, smem, stream>>>(a, static_cast<int>(rows), vec_out, z0);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  const int n_red = a.op == 0 ? a.C : a.K;
  const int n_out = a.op == 0 ? a.K : a.C;
  const bool v = vec && n_red % 4 == 0 && (a.op == 0 || n_out % 4 == 0);
  if (a.op == 0) return v ? pick_fwd<true, true>(a, n_red, n_out, num_sms, stream) : pick_fwd<true, false>(a, n_red, n_out, num_sms, stream);
  return v ? pick_fwd<false, true>(a, n_red, n_out, num_sms, stream) : pick_fwd<false, false>(a, n_red, n_out, num_sms, stream);
}

}  // namespace scb
