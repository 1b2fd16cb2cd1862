// pairs.cu - indice-pair / mask builder on the GPU.
//
// Replaces spconv's generate_subm_conv_inds / generate_conv_inds and
// sort_1d_by_key_split as they are used by the reference driver
// (cumm/conv/main_real_spconv.py:72-145), over a linear-probing hash table in
// the style of cumm's LinearHashTableSplit (include/tensorview/hash/linear.cu.h:557-840):
// keys are linearised voxel coordinates (int64, empty slot = -1), slot =
// MurmurHash3 64-bit finaliser(key) & (capacity - 1), collisions probe
// linearly.  Unlike the reference's unbounded `while (true)` probe loops
// (linear.cu.h:229,381) every probe here stops after `capacity` steps and
// reports kErrHashFull.
//
// Conventions (cross-correlation, matching torch.nn.functional.conv3d):
//   coords[i] = (batch, z, y, x); offset k = (kz * KY + ky) * KX + kx;
//   submanifold: pairs_fwd[k][i] = index of the voxel at
//     coord(i) + ((kz, ky, kx) - ksize // 2) * dilation, or -1;
//   strided: output o receives input i through offset k iff
//     coord(i) = o * stride - padding + (kz, ky, kx) * dilation;
//   pairs_bwd[k][i] = o such that pairs_fwd[k][o] = i;
//   mask_fwd[o] bit k <=> pairs_fwd[k][o] >= 0; mask_bwd[i] bit k <=> pairs_bwd[k][i] >= 0.
// Strided outputs are numbered in ascending linearised (batch, z, y, x) order
// (the reference numbers them by an atomic counter, i.e. nondeterministically,
// hash.cu.h:201-213; the canonical order makes the table reproducible).
#include "kernels.h"

namespace scb {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ uint64_t fmix64(uint64_t k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return k;
}

struct Table {
  unsigned long long *keys;  // -1 = empty
  int *vals;
  int64_t cap;               // power of two
};

__device__ __forceinline__ bool table_insert(const Table &t, long long key, int val, int *err) {
  uint64_t slot = fmix64(static_cast<uint64_t>(key)) & static_cast<uint64_t>(t.cap - 1);
  for (int64_t step = 0; step < t.cap; ++step) {
    const unsigned long long prev =
        atomicCAS(t.keys + slot, ~0ull, static_cast<unsigned long long>(key));
    if (prev == ~0ull || prev == static_cast<unsigned long long>(key)) {
      if (t.vals) atomicMin(t.vals + slot, val);
      return true;
    }
    slot = (slot + 1) & static_cast<uint64_t>(t.cap - 1);
  }
  atomicOr(err, kErrHashFull);
  return false;
}

__device__ __forceinline__ int table_lookup(const Table &t, long long key) {
  uint64_t slot = fmix64(static_cast<uint64_t>(key)) & static_cast<uint64_t>(t.cap - 1);
  for (int64_t step = 0; step < t.cap; ++step) {
    const unsigned long long k = t.keys[slot];
    if (k == static_cast<unsigned long long>(key)) return t.vals[slot];
    if (k == ~0ull) return -1;
    slot = (slot + 1) & static_cast<uint64_t>(t.cap - 1);
  }
  return -1;
}

__global__ void table_clear(Table t) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < t.cap;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    t.keys[i] = ~0ull;
    if (t.vals) t.vals[i] = 0x7fffffff;
  }
}

struct Geom {
  int spatial[3];
  int ksize[3];
  int stride[3];
  int padding[3];
  int dilation[3];
  int out_spatial[3];
  int kv;
};

__device__ __forceinline__ long long lin_key(int b, int z, int y, int x, const int *sp) {
  return ((static_cast<long long>(b) * sp[0] + z) * sp[1] + y) * sp[2] + x;
}

// ------------------------------------------------------------------ submanifold pairs
// Hash table over groups of four voxels consecutive in x: one 32-byte slot
// (one L2 sector) holds the group's key and the index of each of its voxels
// (-1 = none), so a row of three x-neighbours takes one or two probes instead
// of three.  A group lives in the bucket of eight slots that its hash names
// (where that is full, in the next one with room), and a byte per slot holds
// seven more bits of the hash: a lookup compares a bucket's eight bytes at once
// and reads a slot only where one matches, so absent neighbours (most rows off
// a surface) and other groups' slots cost no slot reads and no probe chains.
// One 0xff fill empties keys, indices and bytes.
struct __align__(32) GroupSlot {
  unsigned long long key;  // ((b * D + z) * H + y) * ceil(W / 4) + x / 4; ~0 = empty
  unsigned long long pad;
  int v[4];
};
struct GroupTable {
  GroupSlot *slot;
  uint8_t *tag;            // 0xff = empty
  int64_t cap;             // power of two, >= 8, > 1.5 x voxels, <= 2^32
  int log2cap;
};

// Groups of a row of w >= 1 voxels (w + 3 may not fit an int).
__device__ __forceinline__ int groups_of(int w) { return ((w - 1) >> 2) + 1; }

// A 32-bit multiplicative hash of the folded key (neighbouring rows and groups
// differ in its low bits, which the multiplications carry to the top): the top
// bits name the slot that an insertion starts at, the low seven are the tag.
// Six instructions: a 64-bit finaliser's twenty were most of the lookups' cost.
__device__ __forceinline__ uint32_t group_hash(unsigned long long key) {
  uint32_t h = static_cast<uint32_t>(key) + static_cast<uint32_t>(key >> 32) * 0x85ebca6bu;
  h *= 0x9e3779b1u;
  h ^= h >> 15;
  return h * 0x2c1b3c6du;
}

// First slot (0..7) of a bucket whose tag matches, -1 if none, with the
// bucket's tags `g`; `open`: the bucket has an empty slot.
__device__ __forceinline__ int match_tags(const uint2 &g, uint32_t hash, bool *open) {
  const uint32_t want = (hash & 127u) * 0x01010101u;
  const uint32_t lo = __vcmpeq4(g.x, want), hi = __vcmpeq4(g.y, want);
  *open = (__vcmpeq4(g.x, 0xffffffffu) | __vcmpeq4(g.y, 0xffffffffu)) != 0u;
  return lo ? (__ffs(lo) - 1) >> 3 : hi ? 4 + ((__ffs(hi) - 1) >> 3) : -1;
}

__device__ __forceinline__ int4 load_coord(const int32_t *coords, int64_t i, bool vec) {
  if (vec) return __ldg(reinterpret_cast<const int4 *>(coords) + i);
  return make_int4(coords[i * 4], coords[i * 4 + 1], coords[i * 4 + 2], coords[i * 4 + 3]);
}

// Lanes of consecutive voxels of one group (their rows are in row order) claim
// their slot once, through the first of them.
__global__ void __launch_bounds__(kThreads)
insert_groups(const int32_t *coords, int vec, int64_t n, Geom g, GroupTable t, int *err) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int4 c = i < n ? load_coord(coords, i, vec != 0) : make_int4(0, 0, 0, 0);
  const bool in = i < n && c.x >= 0 && c.y >= 0 && c.z >= 0 && c.w >= 0 && c.y < g.spatial[0] &&
                  c.z < g.spatial[1] && c.w < g.spatial[2];
  if (i < n && !in) atomicOr(err, kErrBadIndex);
  const int gsp[3] = {g.spatial[0], g.spatial[1], groups_of(g.spatial[2])};
  const unsigned long long key = in ? static_cast<unsigned long long>(lin_key(c.x, c.y, c.z, c.w >> 2, gsp)) : ~0ull;
  const unsigned long long prev_key = __shfl_up_sync(0xffffffffu, key, 1);
  const bool leader = lane == 0 || prev_key != key;
  const uint32_t hash = group_hash(key);
  uint32_t at = hash >> (32 - t.log2cap);
  bool placed = false;
  if (leader && in) {
    // the bucket's eight slots from the hashed one round, then the next bucket
    const uint32_t start = at & 7u;
    uint32_t bucket = at & ~7u;
    for (int64_t step = 0; step < t.cap; ++step) {
      at = bucket | ((start + static_cast<uint32_t>(step)) & 7u);
      const unsigned long long was = atomicCAS(&t.slot[at].key, ~0ull, key);
      placed = was == ~0ull || was == key;
      if (placed) {
        // the tag's byte was 0xff, or holds this tag already
        const uint32_t sh = (at & 3u) * 8u;
        atomicAnd(reinterpret_cast<uint32_t *>(t.tag) + (at >> 2), ~((~hash & 0xffu | 0x80u) << sh));
        break;
      }
      if ((step & 7) == 7) bucket = (bucket + 8u) & static_cast<uint32_t>(t.cap - 1);
    }
    if (!placed) atomicOr(err, kErrHashFull);
  }
  const unsigned leaders = __ballot_sync(0xffffffffu, leader);
  const int src = 31 - __clz(leaders & (0xffffffffu >> (31 - lane)));
  at = __shfl_sync(0xffffffffu, at, src);
  placed = __shfl_sync(0xffffffffu, placed ? 1 : 0, src) != 0;
  // the smallest index of equal coordinates wins (-1 is the largest unsigned)
  if (in && placed)
    atomicMin(reinterpret_cast<unsigned int *>(&t.slot[at].v[c.w & 3]), static_cast<unsigned int>(i));
}

// A slot in one 32-byte load.
__device__ __forceinline__ void load_slot(const GroupSlot *s, unsigned long long &key, int4 &v) {
  unsigned long long pad, lo, hi;
  asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(key), "=l"(pad), "=l"(lo), "=l"(hi) : "l"(s));
  (void)pad;
  v = make_int4(static_cast<int>(lo), static_cast<int>(lo >> 32), static_cast<int>(hi), static_cast<int>(hi >> 32));
}

// The slot of group `key`; null if it is not there.
__device__ __forceinline__ const GroupSlot *find_group(const GroupTable &t, unsigned long long key) {
  const uint32_t hash = group_hash(key);
  const uint32_t want = (hash & 127u) * 0x01010101u;
  uint32_t bucket = (hash >> (32 - t.log2cap)) & ~7u;
  for (int64_t step = 0; step < t.cap; step += 8) {
    const uint2 g = *reinterpret_cast<const uint2 *>(t.tag + bucket);
    for (int half = 0; half < 2; ++half) {
      for (uint32_t m = __vcmpeq4(half ? g.y : g.x, want) & 0x01010101u; m != 0u; m &= m - 1u) {
        const GroupSlot *s = t.slot + bucket + half * 4 + ((__ffs(m) - 1) >> 3);
        if (s->key == key) return s;
      }
    }
    if ((__vcmpeq4(g.x, 0xffffffffu) | __vcmpeq4(g.y, 0xffffffffu)) != 0u) break;
    bucket = (bucket + 8u) & static_cast<uint32_t>(t.cap - 1);
  }
  return nullptr;
}

__device__ __forceinline__ int pick(const int4 &v, int q) {
  const int a = q & 1 ? v.y : v.x, b = q & 1 ? v.w : v.z;
  return q & 2 ? b : a;
}

// Both tables of a submanifold convolution.  Offset k seen from an input is
// offset kv - 1 - k seen from its output, so pairs_bwd[kv - 1 - k][i] is
// pairs_fwd[k][i] and both are written here, coalesced, without a fill and a
// scatter.  A voxel that is not the one the table holds for its coordinates (a
// duplicate, or one outside the grid) is nobody's input: its column of
// pairs_bwd is -1.
//
// 3x3x3, dilation 1 (kNine): per z plane the three rows' probes, and those of
// the second group of lanes at a group's edge, are in flight together.  Bound
// by two dependent round trips per plane (tags, slots) and by its table writes
// (216 bytes per voxel).  Both tables, 200k / 2.6M voxels: 79 / 600 us with 27
// chained hash probes, a fill and a scatter; 25 / 404 with groups and linear
// probing of the slots; 23 / 263 with tags.
template <bool kNine>
__global__ void __launch_bounds__(128)
subm_pairs_kernel(const int32_t *coords, int vec, int64_t n, Geom g, GroupTable t, int32_t *pairs_fwd,
                  int32_t *pairs_bwd, uint32_t *mask_fwd) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const bool live = i < n;
  const int4 co = live ? load_coord(coords, i, vec != 0) : make_int4(0, 0, 0, 0);
  const int z = co.y, y = co.z, x = co.w;
  const int ng = groups_of(g.spatial[2]);
  const int gsp[3] = {g.spatial[0], g.spatial[1], ng};
  uint32_t m = 0;
  if constexpr (kNine) {
    const int q = x & 3;
    const int gx = x >> 2;
    // a lane at its group's edge also wants the neighbour group's voxel next to it
    const int side = q == 0 ? -1 : 1;
    const bool has_main = live && gx >= 0 && gx < ng;
    const bool want_side = (q == 0 || q == 3) && gx + side >= 0 && gx + side < ng;
    const unsigned long long key0 = static_cast<unsigned long long>(lin_key(co.x, z, y, gx, gsp));
    // where the lane beside holds the neighbour group (rows in scan order), its
    // nine probes are this lane's too; both in the grid, as a voxel outside it
    // has the linear key of a group of another row
    const int lane = threadIdx.x & 31;
    const bool inside = live && co.x >= 0 && z >= 0 && y >= 0 && x >= 0 && z < g.spatial[0] && y < g.spatial[1] &&
                        x < g.spatial[2];
    const unsigned long long key_up = __shfl_up_sync(0xffffffffu, key0, 1);
    const unsigned long long key_dn = __shfl_down_sync(0xffffffffu, key0, 1);
    const unsigned in_grid = __ballot_sync(0xffffffffu, inside);
    const int beside = (lane + side) & 31;
    const bool shared = inside && want_side && lane + side == beside && ((in_grid >> beside) & 1u) &&
                        (q == 0 ? key_up == key0 - 1 : key_dn == key0 + 1);
    const bool has_side = live && want_side && !shared;
    const long long dz = static_cast<long long>(g.spatial[1]) * ng;
    __shared__ int sj[27][128];  // [offset][thread]
    const int tid = threadIdx.x;
    // Lookups that a bucket's tags do not settle (a full bucket, two groups with
    // one tag): looked up again after the straight pass, one at a time.
    uint32_t unresolved = 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const bool ok_z = z + a - 1 >= 0 && z + a - 1 < g.spatial[0];
      unsigned long long k_main[3];
      uint32_t h_main[3], h_side[3];
      uint2 g_main[3], g_side[3];
      bool ok[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        ok[c] = ok_z && y + c - 1 >= 0 && y + c - 1 < g.spatial[1];
        const unsigned long long k = key0 + static_cast<unsigned long long>((a - 1) * dz + static_cast<long long>(c - 1) * ng);
        k_main[c] = k;
        h_main[c] = group_hash(k);
        h_side[c] = group_hash(k + static_cast<unsigned long long>(static_cast<long long>(side)));
        g_main[c] = g_side[c] = make_uint2(0xffffffffu, 0xffffffffu);
        if (ok[c] && has_main)
          g_main[c] = __ldg(reinterpret_cast<const uint2 *>(t.tag + ((h_main[c] >> (32 - t.log2cap)) & ~7u)));
        if (ok[c] && has_side)
          g_side[c] = __ldg(reinterpret_cast<const uint2 *>(t.tag + ((h_side[c] >> (32 - t.log2cap)) & ~7u)));
      }
      unsigned long long f_main[3], f_side[3];
      int4 v[3];
      int vs[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        f_main[c] = k_main[c];
        f_side[c] = k_main[c] + static_cast<unsigned long long>(static_cast<long long>(side));
        v[c] = make_int4(-1, -1, -1, -1);
        vs[c] = -1;
        bool open;
        int at = match_tags(g_main[c], h_main[c], &open);
        if (at >= 0)
          load_slot(t.slot + ((h_main[c] >> (32 - t.log2cap)) & ~7u) + at, f_main[c], v[c]);
        else if (!open)
          unresolved |= 1u << (a * 3 + c);
        at = match_tags(g_side[c], h_side[c], &open);
        if (at >= 0) {
          const GroupSlot *s = t.slot + ((h_side[c] >> (32 - t.log2cap)) & ~7u) + at;
          f_side[c] = s->key;
          vs[c] = s->v[side < 0 ? 3 : 0];
        } else if (!open) {
          unresolved |= 512u << (a * 3 + c);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (f_main[c] != k_main[c]) unresolved |= 1u << (a * 3 + c);
        if (f_side[c] != k_main[c] + static_cast<unsigned long long>(static_cast<long long>(side)))
          unresolved |= 512u << (a * 3 + c);
        const int beside_up = __shfl_up_sync(0xffffffffu, v[c].w, 1);
        const int beside_dn = __shfl_down_sync(0xffffffffu, v[c].x, 1);
        if (shared) vs[c] = q == 0 ? beside_up : beside_dn;
        const int k = (a * 3 + c) * 3;
        sj[k][tid] = q == 0 ? vs[c] : pick(v[c], q - 1);
        sj[k + 1][tid] = pick(v[c], q);
        sj[k + 2][tid] = q == 3 ? vs[c] : pick(v[c], q + 1);
      }
    }
    {
      const uint32_t up = __shfl_up_sync(0xffffffffu, unresolved, 1);
      const uint32_t dn = __shfl_down_sync(0xffffffffu, unresolved, 1);
      if (shared) unresolved |= ((q == 0 ? up : dn) & 511u) << 9;
    }
    if (!live) return;
    while (unresolved) {
      const int b = __ffs(unresolved) - 1;
      unresolved &= unresolved - 1u;
      const bool is_side = b >= 9;
      const int r = is_side ? b - 9 : b;
      const unsigned long long key = key0 + static_cast<unsigned long long>(
          (r / 3 - 1) * dz + static_cast<long long>(r % 3 - 1) * ng + (is_side ? side : 0));
      const GroupSlot *s = find_group(t, key);
      if (is_side) {
        sj[r * 3 + (side < 0 ? 0 : 2)][tid] = s ? s->v[side < 0 ? 3 : 0] : -1;
      } else {
        const int4 v = s ? *reinterpret_cast<const int4 *>(s->v) : make_int4(-1, -1, -1, -1);
        if (q > 0) sj[r * 3][tid] = pick(v, q - 1);
        sj[r * 3 + 1][tid] = pick(v, q);
        if (q < 3) sj[r * 3 + 2][tid] = pick(v, q + 1);
      }
    }
    const bool held = sj[13][tid] == static_cast<int>(i);
    int32_t *fwd = pairs_fwd + i;
    int32_t *bwd = pairs_bwd + 26 * n + i;
#pragma unroll
    for (int k = 0; k < 27; ++k, fwd += n, bwd -= n) {
      const int j = sj[k][tid];
      *fwd = j;
      *bwd = held ? j : -1;
      if (j >= 0) m |= 1u << k;
    }
  } else {
    if (!live) return;
    auto lookup = [&](int zz, int yy, int xx) {
      if (zz < 0 || yy < 0 || xx < 0 || zz >= g.spatial[0] || yy >= g.spatial[1] || xx >= g.spatial[2]) return -1;
      const unsigned long long key = static_cast<unsigned long long>(lin_key(co.x, zz, yy, xx >> 2, gsp));
      const GroupSlot *s = find_group(t, key);
      return s ? s->v[xx & 3] : -1;
    };
    const bool held = lookup(z, y, x) == static_cast<int>(i);
    int k = 0;
    for (int a = 0; a < g.ksize[0]; ++a)
      for (int c = 0; c < g.ksize[1]; ++c)
        for (int d = 0; d < g.ksize[2]; ++d, ++k) {
          const int j = lookup(z + (a - g.ksize[0] / 2) * g.dilation[0], y + (c - g.ksize[1] / 2) * g.dilation[1],
                               x + (d - g.ksize[2] / 2) * g.dilation[2]);
          pairs_fwd[static_cast<int64_t>(k) * n + i] = j;
          pairs_bwd[static_cast<int64_t>(g.kv - 1 - k) * n + i] = held ? j : -1;
          if (j >= 0) m |= 1u << k;
        }
  }
  mask_fwd[i] = m;
}

// ------------------------------------------------------------------ strided pairs
// Output coordinate along one axis of input coordinate v through kernel step a; false if none.
__device__ __forceinline__ bool out_axis(const Geom &g, int axis, int v, int a, int &o) {
  const int t = v + g.padding[axis] - a * g.dilation[axis];
  if (t < 0) return false;
  o = t / g.stride[axis];
  return o * g.stride[axis] == t && o < g.out_spatial[axis];
}

// The outputs of one input: calls f(k, o-linear key) for every offset that has
// one, in offset order.  Each axis is divided once per kernel step along it.
template <typename F>
__device__ __forceinline__ void for_each_output(const Geom &g, const int4 &co, F f) {
  for (int a = 0; a < g.ksize[0]; ++a) {
    int oz;
    if (!out_axis(g, 0, co.y, a, oz)) continue;
    for (int c = 0; c < g.ksize[1]; ++c) {
      int oy;
      if (!out_axis(g, 1, co.z, c, oy)) continue;
      for (int d = 0; d < g.ksize[2]; ++d) {
        int ox;
        if (out_axis(g, 2, co.w, d, ox))
          f((a * g.ksize[1] + c) * g.ksize[2] + d, lin_key(co.x, oz, oy, ox, g.out_spatial));
      }
    }
  }
}

// How the outputs of a strided build are held between its two calls.
// Bitmap: one entry per 32 output cells in linear order, so an output's number
// (outputs are numbered in ascending order) is the entry's prefix plus the set
// bits below it: no sort, no hash, one 8-byte load per lookup.  Hash: the key
// table, for grids whose bitmap the workspace cannot hold and for batch
// indices outside the given batch size.
struct BitEntry {
  uint32_t bits, prefix;
};
struct ConvHead {
  int count;     // outputs
  int err;       // the device error word when the count was taken
  int outside;   // a cell lies outside the bitmap: take the hash
  int hash;      // the outputs are held in the hash table
  int done;      // blocks of bitmap_count finished
};

__global__ void bitmap_mark(const int32_t *coords, int vec, int64_t n, Geom g, int64_t cells, BitEntry *map,
                            ConvHead *head) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int4 co = load_coord(coords, i, vec != 0);
  for_each_output(g, co, [&](int, long long o) {
    if (o < 0 || o >= cells) {
      head->outside = 1;
      return;
    }
    atomicOr(&map[o >> 5].bits, 1u << (o & 31));
  });
}

constexpr int kMapThreads = 256;
constexpr int kMapPer = 4;                          // entries per thread
constexpr int kMapBlock = kMapThreads * kMapPer;    // entries per block

__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *total) {
  // exclusive scan over the block's threads (kMapThreads)
  __shared__ uint32_t ws[kMapThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
    if (lane >= s) x += y;
  }
  __syncthreads();
  if (lane == 31) ws[w] = x;
  __syncthreads();
  uint32_t before = 0u, all = 0u;
#pragma unroll
  for (int i = 0; i < kMapThreads / 32; ++i) {
    if (i < w) before += ws[i];
    all += ws[i];
  }
  *total = all;
  return before + x - v;
}

// Set bits per block of entries; the last block to finish turns the block
// counts into their exclusive scan and leaves the total and the error word in
// the head (one copy brings both to the host).
__global__ void __launch_bounds__(kMapThreads)
bitmap_count(const BitEntry *map, int64_t entries, uint32_t *blocks, ConvHead *head, const int *err) {
  const int64_t e0 = static_cast<int64_t>(blockIdx.x) * kMapBlock;
  uint32_t c = 0u;
#pragma unroll
  for (int q = 0; q < kMapPer; ++q) {
    const int64_t e = e0 + q * kMapThreads + threadIdx.x;
    if (e < entries) c += __popc(map[e].bits);
  }
  uint32_t total;
  block_scan(c, &total);
  __shared__ int last;
  if (threadIdx.x == 0) {
    blocks[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(&head->done, 1) == static_cast<int>(gridDim.x) - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  uint32_t carry = 0u;
  for (int64_t b0 = 0; b0 < gridDim.x; b0 += kMapThreads) {
    const int64_t b = b0 + threadIdx.x;
    const uint32_t v = b < gridDim.x ? *reinterpret_cast<volatile uint32_t *>(blocks + b) : 0u;
    uint32_t all;
    const uint32_t x = block_scan(v, &all);
    if (b < gridDim.x) blocks[b] = carry + x;
    carry += all;
  }
  if (threadIdx.x == 0) {
    head->count = static_cast<int>(carry);
    head->err = *err;
    head->hash = 0;
  }
}

__device__ __forceinline__ void store_coord(int32_t *out, int64_t i, bool vec, long long key, const Geom &g) {
  int b, z, y, x;
  if (key < (1ll << 32)) {  // 32-bit divisions
    uint32_t k = static_cast<uint32_t>(key);
    const uint32_t W = g.out_spatial[2], H = g.out_spatial[1], D = g.out_spatial[0];
    x = static_cast<int>(k % W);
    k /= W;
    y = static_cast<int>(k % H);
    k /= H;
    z = static_cast<int>(k % D);
    b = static_cast<int>(k / D);
  } else {
    long long k = key;
    x = static_cast<int>(k % g.out_spatial[2]);
    k /= g.out_spatial[2];
    y = static_cast<int>(k % g.out_spatial[1]);
    k /= g.out_spatial[1];
    z = static_cast<int>(k % g.out_spatial[0]);
    b = static_cast<int>(k / g.out_spatial[0]);
  }
  if (vec) {
    reinterpret_cast<int4 *>(out)[i] = make_int4(b, z, y, x);
  } else {
    out[i * 4] = b;
    out[i * 4 + 1] = z;
    out[i * 4 + 2] = y;
    out[i * 4 + 3] = x;
  }
}

// Prefix of every entry, and the output coordinates in ascending order: a warp
// takes its non-empty entries one by one, lane l bit l.  (Outputs held in the
// hash table: their coordinates only.)
__global__ void __launch_bounds__(kMapThreads)
bitmap_number(BitEntry *map, int64_t entries, const uint32_t *blocks, const unsigned long long *keys,
              const ConvHead *head, Geom g, int64_t n_out, int32_t *out_coords, int vec) {
  if (head->hash) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(kMapThreads) + threadIdx.x; i < n_out;
         i += static_cast<int64_t>(gridDim.x) * kMapThreads)
      store_coord(out_coords, i, vec != 0, static_cast<long long>(keys[i]), g);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t e0 = static_cast<int64_t>(blockIdx.x) * kMapBlock + static_cast<int64_t>(threadIdx.x) * kMapPer;
  uint32_t bits[kMapPer];
  uint32_t c = 0u;
#pragma unroll
  for (int q = 0; q < kMapPer; ++q) {
    bits[q] = e0 + q < entries ? map[e0 + q].bits : 0u;
    c += __popc(bits[q]);
  }
  uint32_t total;
  uint32_t at = blocks[blockIdx.x] + block_scan(c, &total);
  if (total == 0u) return;  // no lookup reads the prefix of an entry without bits
#pragma unroll
  for (int q = 0; q < kMapPer; ++q) {
    if (bits[q]) map[e0 + q].prefix = at;
    for (unsigned some = __ballot_sync(0xffffffffu, bits[q] != 0u); some != 0u; some &= some - 1u) {
      const int src = __ffs(some) - 1;
      const uint32_t m = __shfl_sync(0xffffffffu, bits[q], src);
      const int64_t i = static_cast<int64_t>(__shfl_sync(0xffffffffu, at, src)) + __popc(m & ((1u << lane) - 1u));
      const int64_t e = e0 + q + static_cast<int64_t>(src - lane) * kMapPer;
      if (((m >> lane) & 1u) && i < n_out) store_coord(out_coords, i, vec != 0, e * 32 + lane, g);
    }
    at += __popc(bits[q]);
  }
}

__global__ void conv_candidates(const int32_t *coords, int vec, int64_t n, Geom g, Table t, int *err) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int4 co = load_coord(coords, i, vec != 0);
  for_each_output(g, co, [&](int, long long o) { table_insert(t, o, 0, err); });
}

__global__ void collect_keys(Table t, unsigned long long *out, ConvHead *head) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < t.cap;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const unsigned long long k = t.keys[i];
    if (k != ~0ull) out[atomicAdd(&head->count, 1)] = k;
  }
}

// Sorted keys -> table of output numbers (marks the outputs as held there).
__global__ void insert_keys(const unsigned long long *keys, int64_t n_out, Table t, ConvHead *head, int *err) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i == 0) head->hash = 1;
  if (i < n_out) table_insert(t, static_cast<long long>(keys[i]), static_cast<int>(i), err);
}

// Both tables and both masks.  Bound by its scattered writes and its lookups'
// round trips: 3x3x3 (kNine) takes a z step's nine lookups together.  60k
// voxels, stride 2: 28 us with chained hash lookups and divisions for every
// offset and axis, now 8.
template <bool kNine>
__global__ void __launch_bounds__(128)
conv_pairs_kernel(const int32_t *coords, int vec, int64_t n, int64_t n_out, Geom g, Table t, const BitEntry *map,
                  const ConvHead *head, int32_t *pairs_fwd, int32_t *pairs_bwd, uint32_t *mask_fwd,
                  uint32_t *mask_bwd) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int4 co = load_coord(coords, i, vec != 0);
  const bool hash = head->hash != 0;
  uint32_t m = 0;
  auto number = [&](const uint2 &e, long long key) {
    return static_cast<int>(e.y + __popc(e.x & ((1u << (key & 31)) - 1u)));
  };
  auto put = [&](int k, int o) {
    if (o >= n_out) o = -1;
    pairs_bwd[static_cast<int64_t>(k) * n + i] = o;
    if (o >= 0) {
      m |= 1u << k;
      pairs_fwd[static_cast<int64_t>(k) * n_out + o] = static_cast<int>(i);
      atomicOr(mask_fwd + o, 1u << k);
    }
  };
  if (kNine && !hash) {
    int oy[3], ox[3];
    bool in_y[3], in_x[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      in_y[c] = out_axis(g, 1, co.z, c, oy[c]);
      in_x[c] = out_axis(g, 2, co.w, c, ox[c]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      int oz;
      const bool in_z = out_axis(g, 0, co.y, a, oz);
      uint2 e[9];
      long long key[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const bool ok = in_z && in_y[q / 3] && in_x[q % 3];
        key[q] = ok ? lin_key(co.x, oz, oy[q / 3], ox[q % 3], g.out_spatial) : -1;
        if (ok) e[q] = __ldg(reinterpret_cast<const uint2 *>(map + (key[q] >> 5)));
      }
#pragma unroll
      for (int q = 0; q < 9; ++q) put(a * 9 + q, key[q] >= 0 ? number(e[q], key[q]) : -1);
    }
  } else {
    int k = 0;
    for (int a = 0; a < g.ksize[0]; ++a)
      for (int c = 0; c < g.ksize[1]; ++c)
        for (int d = 0; d < g.ksize[2]; ++d, ++k) {
          int oz, oy, ox;
          int o = -1;
          if (out_axis(g, 0, co.y, a, oz) && out_axis(g, 1, co.z, c, oy) && out_axis(g, 2, co.w, d, ox)) {
            const long long key = lin_key(co.x, oz, oy, ox, g.out_spatial);
            o = hash ? table_lookup(t, key) : number(*reinterpret_cast<const uint2 *>(map + (key >> 5)), key);
          }
          put(k, o);
        }
  }
  mask_bwd[i] = m;
}

// ------------------------------------------------------------------ stable LSD radix sort of strided output keys
// (grids too large for the output bitmap).  8-bit digits; each pass: per-tile digit histograms, one exclusive scan,
// then an order-preserving scatter (tiles of 4096 items, 8 warps x 512).
constexpr int kSortTile = 4096;
constexpr int kSortWarps = 8;

template <typename K>
__global__ void radix_hist(const K *keys, int64_t n, int shift, uint32_t *hist, int nblocks) {
  __shared__ uint32_t h[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kSortTile;
  for (int i = threadIdx.x; i < kSortTile; i += blockDim.x) {
    const int64_t j = base + i;
    if (j < n) atomicAdd(&h[(keys[j] >> shift) & 255u], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    hist[static_cast<int64_t>(i) * nblocks + blockIdx.x] = h[i];
}

// single-block exclusive scan of `n` uint32 in place
__global__ void scan_exclusive(uint32_t *a, int64_t n) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t base = 0; base < n; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    uint32_t v = i < n ? a[i] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
      if (lane >= s) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
      uint32_t ws = lane < static_cast<int>(blockDim.x >> 5) ? warp_sums[lane] : 0u;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, ws, s);
        if (lane >= s) ws += y;
      }
      warp_sums[lane] = ws;
    }
    __syncthreads();
    const uint32_t prefix = (w > 0 ? warp_sums[w - 1] : 0u) + carry;
    if (i < n) a[i] = prefix + x - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = prefix + x;
    __syncthreads();
  }
}

template <typename K>
__global__ void radix_scatter(const K *keys, const int32_t *vals, K *keys_out, int32_t *vals_out,
                              int64_t n, int shift, const uint32_t *hist, int nblocks) {
  __shared__ uint32_t wh[kSortWarps][256];
  __shared__ uint32_t base_off[256];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t tile0 = static_cast<int64_t>(blockIdx.x) * kSortTile;
  const int per_warp = kSortTile / kSortWarps;
  const int64_t w0 = tile0 + static_cast<int64_t>(w) * per_warp;
  for (int i = lane; i < 256; i += 32) wh[w][i] = 0;
  __syncwarp();
  for (int i = lane; i < per_warp; i += 32) {
    const int64_t j = w0 + i;
    if (j < n) atomicAdd(&wh[w][(keys[j] >> shift) & 255u], 1u);
  }
  __syncthreads();
  // exclusive prefix over warps per digit, plus the global base of this tile
  for (int d = threadIdx.x; d < 256; d += blockDim.x) {
    uint32_t run = hist[static_cast<int64_t>(d) * nblocks + blockIdx.x];
    for (int ww = 0; ww < kSortWarps; ++ww) {
      const uint32_t c = wh[ww][d];
      wh[ww][d] = run;
      run += c;
    }
    base_off[d] = 0;
  }
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
  for (int i = 0; i < per_warp; i += 32) {
    const int64_t j = w0 + i + lane;
    const bool v = j < n;
    const uint32_t d = v ? static_cast<uint32_t>((keys[j] >> shift) & 255u) : 256u + lane;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const uint32_t rank = __popc(peers & lt);
    uint32_t pos = 0;
    if (v) pos = wh[w][d] + rank;
    __syncwarp();
    if (v && rank == 0) wh[w][d] += __popc(peers);
    __syncwarp();
    if (v) {
      keys_out[pos] = keys[j];
      vals_out[pos] = vals[j];
    }
  }
}

// ------------------------------------------------------------------ stable LSD sort of the mask words
// Digits of up to 8 bits over the set range of the split mask.  A key keeps its
// full mask word through every pass (the digit masks it), and the row number
// is implicit in the first pass, so the last pass writes the sorted masks and
// the argsort themselves.  One launch per pass: a tile's destination offsets
// are the digit's base (digit totals do not change between passes, so
// mask_count_kernel takes those of every pass at once) plus the counts of the
// tiles before it, which each pass leaves for the next one with reductions
// (the key's destination names its next tile).  Bound: launches and dependent
// memory round trips.  Above kMaskRowTiles tiles the counts are taken by their
// own launch and scanned by another: there the reductions cost more than those
// (2.6M rows: 43 us a pass with them, 23 + 9 + 4 without).
// Per pass, against a histogram, a one-block scan and a match_any scatter:
// 200k rows 36 -> 10 us, 60k rows 26 -> 5, 2.6M rows 148 -> 36.
constexpr int kMaskThreads = 256;
constexpr int kMaskWarps = kMaskThreads / 32;
constexpr int kMaskBins = 256;
constexpr int kMaskPasses = 4;
// Up to this many tiles a tile sums the counts before it itself (one short row per digit).
constexpr int kMaskRowTiles = 256;
// Up to this many rows tiles have 1024 of them, above 2048.
constexpr int64_t kMaskSmallRows = (int64_t(kMaskRowTiles) << 10) / 2;

struct MaskSort {
  int64_t n;
  uint32_t split;      // split mask
  int lo, bits;        // first digit: (key & split) >> lo, `bits` bits
  int passes;
  int tile_shift;      // rows per tile = 1 << tile_shift
  int tiles, pitch;    // row tiles, count row pitch (multiple of 4)
};

// Counts of digit p0 per tile, and (totals given) of every pass's digits over all rows.
__global__ void __launch_bounds__(kMaskThreads)
mask_count_kernel(const uint32_t *keys, MaskSort P, int p0, uint32_t *count, uint32_t *totals) {
  __shared__ uint32_t h[kMaskPasses][kMaskBins];
  for (int i = threadIdx.x; i < kMaskPasses * kMaskBins; i += kMaskThreads) h[0][i] = 0u;
  __syncthreads();
  const int64_t base = static_cast<int64_t>(blockIdx.x) << P.tile_shift;
  const uint32_t dm = (1u << P.bits) - 1u;
  for (int i = threadIdx.x; i < (1 << P.tile_shift); i += kMaskThreads) {
    const int64_t j = base + i;
    const bool v = j < P.n;
    const uint32_t key = v ? (keys[j] & P.split) >> P.lo : 0u;
    for (int p = 0; p < P.passes; ++p)
      if (v && (p == p0 || totals != nullptr)) atomicAdd(&h[p][(key >> (p * P.bits)) & dm], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d <= static_cast<int>(dm); d += kMaskThreads) {
    count[static_cast<int64_t>(d) * P.pitch + blockIdx.x] = h[p0][d];
    for (int p = 0; p < P.passes; ++p)
      if (totals != nullptr && h[p][d]) atomicAdd(totals + p * kMaskBins + d, h[p][d]);
  }
}

// Exclusive scan of every digit's row of tile counts (grid: one block per digit).
__global__ void __launch_bounds__(kMaskThreads) mask_rowscan_kernel(uint32_t *count, MaskSort P) {
  __shared__ uint32_t warp_sum[kMaskWarps];
  uint32_t *row = count + static_cast<int64_t>(blockIdx.x) * P.pitch;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t carry = 0u;
  for (int t0 = 0; t0 < P.tiles; t0 += kMaskThreads) {
    const int t = t0 + threadIdx.x;
    const uint32_t v = t < P.tiles ? row[t] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
      if (lane >= s) x += y;
    }
    if (lane == 31) warp_sum[w] = x;
    __syncthreads();
    uint32_t before = carry, all = 0u;
#pragma unroll
    for (int i = 0; i < kMaskWarps; ++i) {
      if (i < w) before += warp_sum[i];
      all += warp_sum[i];
    }
    if (t < P.tiles) row[t] = before + x - v;
    carry += all;
    __syncthreads();
  }
}

// One stable pass.  kItems rows per thread, 32 * kItems consecutive rows per warp.
// vals_in null: row j carries value j.  scanned: count rows hold exclusive sums.
template <int kItems>
__global__ void __launch_bounds__(kMaskThreads)
mask_scatter_kernel(const uint32_t *keys_in, const int32_t *vals_in, uint32_t *keys_out, int32_t *vals_out,
                    MaskSort P, int pass, int scanned, const uint32_t *count, const uint32_t *totals,
                    uint32_t *count_next) {
  __shared__ uint32_t wh[kMaskWarps][kMaskBins];
  __shared__ uint32_t before[kMaskThreads];
  __shared__ uint32_t warp_sum[kMaskWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int tile = blockIdx.x;
  const int bins = 1 << P.bits;
  const int shift = P.lo + pass * P.bits;
  const uint32_t dm = static_cast<uint32_t>(bins) - 1u;
  const int64_t j0 = (static_cast<int64_t>(tile) << P.tile_shift) + w * 32 * kItems + lane;
  uint32_t key[kItems];
  int32_t val[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int64_t j = j0 + i * 32;
    key[i] = j < P.n ? keys_in[j] : 0u;
    val[i] = j < P.n ? (vals_in ? vals_in[j] : static_cast<int32_t>(j)) : 0;
  }
  for (int d = lane; d < bins; d += 32) wh[w][d] = 0u;
  // digit bases: exclusive scan of the totals, plus the tiles before this one
  {
    const int d = threadIdx.x;
    const uint32_t v = d < bins ? totals[pass * kMaskBins + d] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
      if (lane >= s) x += y;
    }
    if (lane == 31) warp_sum[w] = x;
    before[d] = 0u;
    __syncthreads();
    uint32_t base = x - v;
    for (int i = 0; i < w; ++i) base += warp_sum[i];
    if (scanned) {
      if (d < bins) before[d] = base + count[static_cast<int64_t>(d) * P.pitch + tile];
    } else {
      // kMaskThreads / bins threads per digit, each every 4th group of 4 tiles
      const int per = kMaskThreads / bins;
      const int dd = threadIdx.x / per, part = threadIdx.x % per;
      const uint4 *row = reinterpret_cast<const uint4 *>(count + static_cast<int64_t>(dd) * P.pitch);
      uint32_t sum = 0u;
#pragma unroll 8
      for (int q = part; q * 4 < tile; q += per) {
        const uint4 c = row[q];
        const int t = q * 4;
        sum += c.x + (t + 1 < tile ? c.y : 0u) + (t + 2 < tile ? c.z : 0u) + (t + 3 < tile ? c.w : 0u);
      }
      if (d < bins) atomicAdd(&before[d], base);
      if (sum) atomicAdd(&before[dd], sum);
    }
  }
  // rank of every row among the warp's rows of the same digit
  uint16_t rank[kItems];
  const unsigned lt = (1u << lane) - 1u;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const bool v = j0 + i * 32 < P.n;
    const uint32_t d = ((key[i] & P.split) >> shift) & dm;
    unsigned peers = __ballot_sync(0xffffffffu, v);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const unsigned set = __ballot_sync(0xffffffffu, (d >> b) & 1u);
      peers &= ((d >> b) & 1u) ? set : ~set;
    }
    const uint32_t r = __popc(peers & lt);
    const uint32_t at = v ? wh[w][d] : 0u;
    rank[i] = static_cast<uint16_t>(at + r);
    __syncwarp();
    if (v && r == 0u) wh[w][d] = at + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x < bins) {
    uint32_t run = before[threadIdx.x];
#pragma unroll
    for (int i = 0; i < kMaskWarps; ++i) {
      const uint32_t c = wh[i][threadIdx.x];
      wh[i][threadIdx.x] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const bool v = j0 + i * 32 < P.n;
    const uint32_t masked = (key[i] & P.split) >> shift;
    const uint32_t pos = wh[w][masked & dm] + rank[i];
    if (v) {
      keys_out[pos] = key[i];
      vals_out[pos] = val[i];
    }
    if (count_next != nullptr) {
      // Equal masks come in runs and end in one tile: one reduction per
      // distinct counter of the warp.  (One per key met at the same few lines
      // of the counts: 84 us a pass at 1M rows.)
      const uint32_t next = (masked >> P.bits) & dm, to = pos >> P.tile_shift;
      const unsigned peers = __match_any_sync(0xffffffffu, v ? (next << 24 | to) : 0xffffffffu);
      if (v && (peers & lt) == 0u)
        atomicAdd(count_next + static_cast<int64_t>(next) * P.pitch + to, static_cast<uint32_t>(__popc(peers)));
    }
  }
}

MaskSort mask_sort_plan(int64_t n, uint32_t split) {
  MaskSort P{};
  P.n = n;
  P.split = split;
  P.lo = split ? __builtin_ctz(split) : 0;
  const int bits = split ? 32 - __builtin_clz(split) - P.lo : 1;
  P.passes = (bits + 7) / 8;
  P.bits = (bits + P.passes - 1) / P.passes;
  // Small tiles while that keeps the count rows short: more blocks, fewer
  // serial rounds per warp, against more rows for every tile to sum (200k rows
  // a pass: 11.3 us with 196 tiles, 10.1 with 98).
  P.tile_shift = n <= kMaskSmallRows ? 10 : 11;
  P.tiles = static_cast<int>((n + (int64_t(1) << P.tile_shift) - 1) >> P.tile_shift);
  P.pitch = (P.tiles + 3) & ~3;
  return P;
}

__global__ void iota_kernel(int32_t *p, int64_t n) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    p[i] = static_cast<int32_t>(i);
}

inline int grid_for(int64_t n) {
  int64_t b = (n + kThreads - 1) / kThreads;
  if (b > 65535) b = 65535;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

int64_t align_up(int64_t x) { return (x + 255) & ~static_cast<int64_t>(255); }
uint8_t *align_ptr(void *p) {
  return reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(p) + 255) & ~static_cast<uintptr_t>(255));
}

int64_t radix_ws_bytes(int64_t n, int key_bytes) {
  const int64_t nblocks = (n + kSortTile - 1) / kSortTile;
  return align_up(n * key_bytes) + align_up(n * 4) + align_up(256 * nblocks * 4);
}

// Sorts (keys, vals) stably by the low `bits` bits of the keys.  The sorted
// result ends in (keys, vals) again.  ws: radix_ws_bytes(n, sizeof(K)).
template <typename K>
cudaError_t radix_sort(K *keys, int32_t *vals, int64_t n, int bits, uint8_t *ws,
                       cudaStream_t s) {
  if (n <= 1) return cudaSuccess;
  const int nblocks = static_cast<int>((n + kSortTile - 1) / kSortTile);
  K *k2 = reinterpret_cast<K *>(ws);
  int32_t *v2 = reinterpret_cast<int32_t *>(ws + align_up(n * sizeof(K)));
  uint32_t *hist = reinterpret_cast<uint32_t *>(ws + align_up(n * sizeof(K)) + align_up(n * 4));
  K *src_k = keys, *dst_k = k2;
  int32_t *src_v = vals, *dst_v = v2;
  int passes = (bits + 7) / 8;
  if (passes < 1) passes = 1;
  for (int p = 0; p < passes; ++p) {
    const int shift = 8 * p;
    radix_hist<K><<<nblocks, 256, 0, s>>>(src_k, n, shift, hist, nblocks);
    scan_exclusive<<<1, 1024, 0, s>>>(hist, static_cast<int64_t>(256) * nblocks);
    radix_scatter<K><<<nblocks, 32 * kSortWarps, 0, s>>>(src_k, src_v, dst_k, dst_v, n, shift,
                                                         hist, nblocks);
    K *tk = src_k; src_k = dst_k; dst_k = tk;
    int32_t *tv = src_v; src_v = dst_v; dst_v = tv;
  }
  if (src_k != keys) {
    cudaMemcpyAsync(keys, src_k, n * sizeof(K), cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(vals, src_v, n * 4, cudaMemcpyDeviceToDevice, s);
  }
  return cudaGetLastError();
}

int64_t next_pow2(int64_t x) {
  int64_t p = 1;
  while (p < x) p <<= 1;
  return p;
}

Geom make_geom(const PairBuildArgs &a) {
  Geom g;
  for (int d = 0; d < 3; ++d) {
    g.spatial[d] = a.spatial[d];
    g.ksize[d] = a.ksize[d];
    g.stride[d] = a.stride[d];
    g.padding[d] = a.padding[d];
    g.dilation[d] = a.dilation[d];
    g.out_spatial[d] = a.out_spatial[d];
  }
  g.kv = a.ksize[0] * a.ksize[1] * a.ksize[2];
  return g;
}

struct ConvWs {
  ConvHead *head;
  BitEntry *map;               // bitmap entries, then its block counts
  uint32_t *blocks;
  Table set;                   // output key set (no values), later output index table
  unsigned long long *ukeys;   // unique keys
  int32_t *uvals;
  uint8_t *sort_ws;
};

int64_t hash_bytes(int64_t n_in, int kv) {
  // kv bounds outputs_per_input from above
  const int64_t max_out = n_in * kv;
  const int64_t cap = next_pow2(2 * (max_out > 0 ? max_out : 1));
  return align_up(cap * 8) + align_up(cap * 4) + align_up(max_out * 8) + align_up(max_out * 4) +
         radix_ws_bytes(max_out, 8);
}

// A strided workspace holds the hash route, and at least this much, so that
// the bitmap of a 67M-cell output grid fits whatever the voxel count.
constexpr int64_t kMinMapBytes = int64_t(16) << 20;
int64_t conv_bytes(int64_t n_in, int kv) {
  const int64_t h = hash_bytes(n_in, kv);
  return h > kMinMapBytes ? h : kMinMapBytes;
}

int64_t group_cap(int64_t n) { return next_pow2(n + n / 2 + 8); }

int64_t map_cells(const Geom &g, int64_t batch) {
  const double est = static_cast<double>(batch) * g.out_spatial[0] * g.out_spatial[1] * g.out_spatial[2];
  if (est > 1e15) return int64_t(1) << 50;
  return batch * g.out_spatial[0] * g.out_spatial[1] * g.out_spatial[2];
}
int64_t map_entries(int64_t cells) { return (cells + 31) / 32; }
int64_t map_blocks(int64_t cells) { return (map_entries(cells) + kMapBlock - 1) / kMapBlock; }
// The bitmap is cleared, counted and numbered at HBM rate (24 bytes per 32
// cells); the hash route costs a 12-byte slot per possible output twice and a
// sort.  With the workspace as the limit a voxel may have up to ~10k cells.
// 60k voxels in a 21 x 800 x 704 output grid: the outputs in order take 145 us
// with the hash, 23 us with the bitmap.
bool map_fits(int64_t cells, int64_t n_in, int kv) {
  return cells > 0 && align_up(map_entries(cells) * 8) + align_up(map_blocks(cells) * 4) <= conv_bytes(n_in, kv);
}

}  // namespace

int64_t pairs_workspace_bytes(int64_t n_in, int kv, int subm) {
  // 512: the head of a strided build and the alignment of the pointer given
  if (subm) return group_cap(n_in) * (static_cast<int64_t>(sizeof(GroupSlot)) + 1) + 512;
  return conv_bytes(n_in, kv) + 512;
}

static ConvWs carve_conv_ws(void *ws, int64_t n_in, int kv, int64_t cells) {
  ConvWs w;
  const int64_t max_out = n_in * kv;
  const int64_t cap = next_pow2(2 * (max_out > 0 ? max_out : 1));
  uint8_t *p = align_ptr(ws);
  w.head = reinterpret_cast<ConvHead *>(p);
  p += 256;
  w.map = reinterpret_cast<BitEntry *>(p);
  w.blocks = reinterpret_cast<uint32_t *>(p + align_up(map_entries(cells) * 8));
  w.set.keys = reinterpret_cast<unsigned long long *>(p);
  p += align_up(cap * 8);
  w.set.vals = reinterpret_cast<int *>(p);
  p += align_up(cap * 4);
  w.set.cap = cap;
  w.ukeys = reinterpret_cast<unsigned long long *>(p);
  p += align_up(max_out * 8);
  w.uvals = reinterpret_cast<int32_t *>(p);
  p += align_up(max_out * 4);
  w.sort_ws = p;
  return w;
}

static int blocks_of(int64_t n, int threads) { return static_cast<int>((n + threads - 1) / threads); }

cudaError_t build_subm_pairs(const PairBuildArgs &a, int32_t *pairs_fwd, int32_t *pairs_bwd,
                             uint32_t *mask_fwd, void *ws, int64_t ws_bytes, cudaStream_t s) {
  const Geom g = make_geom(a);
  const int64_t n = a.n_in;
  if (n == 0) return cudaSuccess;
  if (ws_bytes < pairs_workspace_bytes(n, g.kv, 1)) return cudaErrorInvalidValue;
  GroupTable t;
  t.cap = group_cap(n);
  t.log2cap = 63 - __builtin_clzll(static_cast<unsigned long long>(t.cap));
  t.slot = reinterpret_cast<GroupSlot *>(align_ptr(ws));
  const int vec = reinterpret_cast<uintptr_t>(a.coords) % 16 == 0;
  t.tag = reinterpret_cast<uint8_t *>(t.slot + t.cap);
  cudaError_t e = cudaMemsetAsync(t.slot, 0xff, t.cap * (sizeof(GroupSlot) + 1), s);
  if (e != cudaSuccess) return e;
  insert_groups<<<blocks_of(n, kThreads), kThreads, 0, s>>>(a.coords, vec, n, g, t, a.err);
  bool nine = true;
  for (int d = 0; d < 3; ++d) nine = nine && g.ksize[d] == 3 && g.dilation[d] == 1;
  (nine ? subm_pairs_kernel<true> : subm_pairs_kernel<false>)<<<blocks_of(n, 128), 128, 0, s>>>(
      a.coords, vec, n, g, t, pairs_fwd, pairs_bwd, mask_fwd);
  return cudaGetLastError();
}

// The count and error word of the head, on the host.
static cudaError_t read_head(const ConvWs &w, ConvHead *h, cudaStream_t s) {
  cudaError_t e = cudaMemcpyAsync(h, w.head, sizeof(ConvHead), cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(s);
}

cudaError_t build_conv_outputs(const PairBuildArgs &a, int64_t *n_out, int *err_bits, void *ws, int64_t ws_bytes,
                               cudaStream_t s) {
  const Geom g = make_geom(a);
  const int64_t n = a.n_in;
  *n_out = 0;
  *err_bits = 0;
  cudaError_t e;
  if (n == 0) {
    e = cudaMemcpyAsync(err_bits, a.err, sizeof(int), cudaMemcpyDeviceToHost, s);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
  }
  if (ws_bytes < pairs_workspace_bytes(n, g.kv, 0)) return cudaErrorInvalidValue;
  const int64_t cells = map_cells(g, a.batch);
  const ConvWs w = carve_conv_ws(ws, n, g.kv, cells);
  const int vec = reinterpret_cast<uintptr_t>(a.coords) % 16 == 0;
  ConvHead h{};
  if (map_fits(cells, n, g.kv)) {
    // the head and the entries in one fill
    e = cudaMemsetAsync(w.head, 0, 256 + map_entries(cells) * 8, s);
    if (e != cudaSuccess) return e;
    bitmap_mark<<<blocks_of(n, 128), 128, 0, s>>>(a.coords, vec, n, g, cells, w.map, w.head);
    bitmap_count<<<static_cast<unsigned>(map_blocks(cells)), kMapThreads, 0, s>>>(w.map, map_entries(cells), w.blocks,
                                                                                  w.head, a.err);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = read_head(w, &h, s);
    if (e != cudaSuccess) return e;
    if (!h.outside) {
      *n_out = h.count;
      *err_bits = h.err;
      return cudaSuccess;
    }
  }
  Table set = w.set;
  e = cudaMemsetAsync(w.head, 0, 256, s);
  if (e != cudaSuccess) return e;
  table_clear<<<grid_for(set.cap), kThreads, 0, s>>>(set);
  Table keys_only = set;
  keys_only.vals = nullptr;
  conv_candidates<<<blocks_of(n, 128), 128, 0, s>>>(a.coords, vec, n, g, keys_only, a.err);
  collect_keys<<<grid_for(set.cap), kThreads, 0, s>>>(set, w.ukeys, w.head);
  e = read_head(w, &h, s);
  if (e != cudaSuccess) return e;
  const long long total = static_cast<long long>(a.batch) * g.out_spatial[0] * g.out_spatial[1] *
                          g.out_spatial[2];
  int bits = 1;
  while (bits < 63 && (1ll << bits) < total) ++bits;
  iota_kernel<<<grid_for(h.count), kThreads, 0, s>>>(w.uvals, h.count);
  e = radix_sort<unsigned long long>(w.ukeys, w.uvals, h.count, bits, w.sort_ws, s);
  if (e != cudaSuccess) return e;
  table_clear<<<grid_for(set.cap), kThreads, 0, s>>>(set);
  insert_keys<<<blocks_of(h.count > 0 ? h.count : 1, kThreads), kThreads, 0, s>>>(w.ukeys, h.count, set, w.head,
                                                                                  a.err);
  *n_out = h.count;
  e = cudaMemcpyAsync(err_bits, a.err, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(s);
}

cudaError_t build_conv_pairs(const PairBuildArgs &a, int64_t n_out, int32_t *out_coords,
                             int32_t *pairs_fwd, int32_t *pairs_bwd, uint32_t *mask_fwd,
                             uint32_t *mask_bwd, void *ws, int64_t ws_bytes, cudaStream_t s) {
  const Geom g = make_geom(a);
  const int64_t n = a.n_in;
  if (n == 0) return cudaSuccess;
  if (ws_bytes < pairs_workspace_bytes(n, g.kv, 0)) return cudaErrorInvalidValue;
  const int64_t cells = map_cells(g, a.batch);
  const ConvWs w = carve_conv_ws(ws, n, g.kv, cells);
  const int vec = reinterpret_cast<uintptr_t>(a.coords) % 16 == 0;
  const int vec_out = reinterpret_cast<uintptr_t>(out_coords) % 16 == 0;
  if (n_out > 0) {
    cudaError_t e = cudaMemsetAsync(pairs_fwd, 0xff, n_out * g.kv * 4, s);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(mask_fwd, 0, n_out * 4, s);
    if (e != cudaSuccess) return e;
    const int64_t blocks = map_fits(cells, n, g.kv) ? map_blocks(cells) : blocks_of(n_out, kMapThreads);
    bitmap_number<<<static_cast<unsigned>(blocks), kMapThreads, 0, s>>>(w.map, map_entries(cells), w.blocks, w.ukeys,
                                                                       w.head, g, n_out, out_coords, vec_out);
  }
  const bool nine = g.ksize[0] == 3 && g.ksize[1] == 3 && g.ksize[2] == 3;
  (nine ? conv_pairs_kernel<true> : conv_pairs_kernel<false>)<<<blocks_of(n, 128), 128, 0, s>>>(
      a.coords, vec, n, n_out, g, w.set, w.map, w.head, pairs_fwd, pairs_bwd, mask_fwd, mask_bwd);
  return cudaGetLastError();
}

namespace {
// One row per thread, kSortOffsets offsets per block row: their loads are in
// flight together.  Bound by L2 throughput of the gathers' sectors (79 % of
// its peak at 1M rows; 75 % of the fetched bytes are not wanted), so an offset
// whose bit the row's mask does not have (given: about half of them) is not
// read.  27 offsets: 200k rows 25 us with one element per thread and a 64-bit
// division each, 22 without the masks, 14 with; 2.6M rows 277, 270, 168.
constexpr int kSortOffsets = 9;
__global__ void __launch_bounds__(kThreads)
sort_indices_kernel(const int32_t *indices, int kv, int64_t n, const int32_t *argsort, const uint32_t *mask,
                    int reverse, int32_t *out) {
  const int64_t r = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x;
  if (r >= n) return;
  const int sig = argsort[r];
  uint32_t m = mask != nullptr ? mask[r] : 0xffffffffu;
  if (reverse) m = __brev(m) >> (32 - kv);
  if (sig < 0 || sig >= n) m = 0u;
  const int k0 = blockIdx.y * kSortOffsets;
  int v[kSortOffsets];
#pragma unroll
  for (int q = 0; q < kSortOffsets; ++q)
    v[q] = k0 + q < kv && ((m >> (k0 + q)) & 1u) ? __ldg(indices + (k0 + q) * n + sig) : -1;
#pragma unroll
  for (int q = 0; q < kSortOffsets; ++q)
    if (k0 + q < kv) out[(k0 + q) * n + r] = v[q];
}
}  // namespace

cudaError_t sort_indices(const int32_t *indices, int kv, int64_t n, const int32_t *argsort,
                         const uint32_t *mask, int reverse, int32_t *out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const dim3 grid(static_cast<unsigned>(blocks_of(n, kThreads)), (kv + kSortOffsets - 1) / kSortOffsets);
  sort_indices_kernel<<<grid, kThreads, 0, s>>>(indices, kv, n, argsort, mask, reverse, out);
  return cudaGetLastError();
}

// Never less for more rows (a workspace is often sized once, for the largest
// call): just above kMaskSmallRows there are fewer tiles, so the counts of the
// small tiles are what is asked for.
int64_t sort_workspace_bytes(int64_t n) {
  if (n <= 0) return 0;
  int64_t pitch = mask_sort_plan(n, 0xffffffffu).pitch;
  if (n > kMaskSmallRows) {
    const int64_t small = mask_sort_plan(kMaskSmallRows, 0xffffffffu).pitch;
    pitch = pitch > small ? pitch : small;
  }
  return 3 * align_up(n * 4) + align_up((pitch + 1) * kMaskPasses * kMaskBins * 4) + 256;
}

cudaError_t sort_masks_split(uint32_t *data, int64_t n, uint32_t split_mask, int32_t *argsort,
                             void *ws, int64_t ws_bytes, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (ws_bytes < sort_workspace_bytes(n)) return cudaErrorInvalidValue;
  const MaskSort P = mask_sort_plan(n, split_mask);
  uint8_t *p = align_ptr(ws);
  uint32_t *ka = reinterpret_cast<uint32_t *>(p);
  int32_t *va = reinterpret_cast<int32_t *>(p + align_up(n * 4));
  uint32_t *kb = reinterpret_cast<uint32_t *>(p + 2 * align_up(n * 4));
  uint32_t *totals = reinterpret_cast<uint32_t *>(p + 3 * align_up(n * 4));
  uint32_t *counts = totals + kMaskPasses * kMaskBins;
  const int64_t per_pass = static_cast<int64_t>(P.pitch) << P.bits;
  cudaError_t e = cudaMemsetAsync(totals, 0, (kMaskPasses * kMaskBins + P.passes * per_pass) * 4, s);
  if (e != cudaSuccess) return e;
  mask_count_kernel<<<P.tiles, kMaskThreads, 0, s>>>(data, P, 0, counts, totals);
  const int scanned = P.tiles > kMaskRowTiles ? 1 : 0;
  const uint32_t *src_k = data;
  const int32_t *src_v = nullptr;
  for (int pass = 0; pass < P.passes; ++pass) {
    // the last pass reads (ka, va) and writes (data, argsort); the passes
    // before it alternate between (ka, va) and (kb, argsort)
    const bool last = pass == P.passes - 1;
    const bool to_a = ((P.passes - 1 - pass) & 1) != 0;
    uint32_t *dst_k = last ? (P.passes > 1 ? data : ka) : to_a ? ka : kb;
    int32_t *dst_v = to_a ? va : argsort;
    uint32_t *count = counts + pass * per_pass;
    uint32_t *next = last || scanned ? nullptr : count + per_pass;
    if (scanned && pass > 0) mask_count_kernel<<<P.tiles, kMaskThreads, 0, s>>>(src_k, P, pass, count, nullptr);
    if (scanned) mask_rowscan_kernel<<<1 << P.bits, kMaskThreads, 0, s>>>(count, P);
    if (P.tile_shift == 10)
      mask_scatter_kernel<4><<<P.tiles, kMaskThreads, 0, s>>>(src_k, src_v, dst_k, dst_v, P, pass, scanned, count,
                                                              totals, next);
    else
      mask_scatter_kernel<8><<<P.tiles, kMaskThreads, 0, s>>>(src_k, src_v, dst_k, dst_v, P, pass, scanned, count,
                                                              totals, next);
    src_k = dst_k;
    src_v = dst_v;
  }
  if (P.passes == 1) cudaMemcpyAsync(data, ka, n * 4, cudaMemcpyDeviceToDevice, s);
  return cudaGetLastError();
}

}  // namespace scb
