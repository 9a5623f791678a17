// gbx_join_packed.cu -- hash joins whose key packs into one 64-bit word
// (fixed-width columns of at most 64 bits together, null bits included).
//
// The general join (gbx_join.cu) stores build *row indices* in its table, so
// a probe reads a slot, then the build key that row names: two dependent
// random reads a probe, through the generic leaf comparison.  Here a 16-byte
// slot holds the packed key itself beside the key's row count and a build
// row of it, so a probe row is one 32-byte load in the usual case, from L2 where
// the table fits (32 MB for 1M build rows).  A thread keeps kJFlight loads in
// flight; the probe is still bound by their latency: 76 registers allow 24
// warps an SM, and lanes that are done leave 14 of 32 active an instruction
// (20M probe rows: L2 at 29% of its peak, DRAM at 12%, issue at 37%).
//
// The output is sized per tile of kJTile probe rows (a 64-bit count per tile
// and a scan over the tiles) instead of per probe row, so the pass between
// finding and writing moves 4 bytes a probe row (the matched build row, or
// the matched slot when some build key repeats) instead of 20.
//
// Measured on B200, 50M probe rows against 1M unique int64 keys: the general
// path's probe 2,056 us, scan 232 us, emit 443 us; here probe 647 us, scan
// 8 us, emit 88 us (and with one 16-byte slot a load instead of a sector of
// two: probe 861 us; with the rows of a thread resolved one after another:
// 966 us).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "../../include/gbx.h"
#include "gbx_device.cuh"
#include "gbx_host.hpp"
#include "gbx_join.hpp"
#include "gbx_scan.hpp"

namespace gbx {

using namespace dev;

namespace {

constexpr int32_t kJoinNoneValue = INT32_MIN;  // cudf::JoinNoneValue (join.hpp)
constexpr int kJBlock            = 256;
constexpr int kJPer              = 8;  // probe rows of a thread
constexpr int kJFlight           = 4;  // of which so many probe at a time
constexpr int kJTile             = kJBlock * kJPer;
constexpr uint32_t kNoSlot       = 0xffffffffu;
// outputs of a block of k_pjoin_emit_runs: enough that the scan of its tile's
// rows (2,048 lookups in the table) stays a small part of the work, or as few
// as kEmitLeast while there are not two blocks an SM
constexpr int64_t kEmitPart  = 32768;
constexpr int64_t kEmitLeast = 2048;
constexpr uintptr_t kSectorBytes = 32;  // a load_sector, aligned
// build rows up to which a slot index and a representative (the reserved
// slot's included) stay below kNoSlot
constexpr int64_t kMaxBuildRows = int64_t(1) << 30;

// One key of the build side: `first` is a build row of it, the key's
// representative (any one of its rows).  The all-ones word marks an
// empty slot; a key of all ones has the reserved slot `cap` (and the
// representative `n`, one past the build rows, since its slot is not claimed
// by a compare-and-swap).  Slots are probed in pairs, each pair one
// 32-byte sector: a key's home is a sector, and a probe examines a sector per
// load (1.1 sectors a probe on average at the loads used, against 1.6 with
// single slots).
struct alignas(16) Slot {
  unsigned long long key;
  uint32_t cnt;
  uint32_t first;
};

struct PackedTable {
  Slot* slots;    // cap + 1
  uint64_t cap;   // power of two
  uint32_t* dup;  // 1 when some build key repeats
};

// Packed key of row r; false when the row matches nothing (a null key under
// null_equality::UNEQUAL).  KM 1 / 2: a single plain 8- / 4-byte column, whose
// bits are the key (no per-column loop).
template <int KM>
__device__ __forceinline__ bool row_key(const KeyPlan& kp, int64_t r, uint64_t& k)
{
  if constexpr (KM == 1) {
    k = __ldg(reinterpret_cast<const unsigned long long*>(kp.cols[0].data) + kp.cols[0].offset + r);
    return true;
  } else if constexpr (KM == 2) {
    k = __ldg(reinterpret_cast<const uint32_t*>(kp.cols[0].data) + kp.cols[0].offset + r);
    return true;
  } else {
    uint64_t kk[1];
    const bool kept = pack_key<1>(kp, r, kk);
    k               = kk[0];
    return kept;
  }
}

// Both slots of sector b (a 32-byte load).
struct Sector {
  unsigned long long key[2];
  uint32_t cnt[2];
  uint32_t first[2];
};
__device__ __forceinline__ Sector load_sector(const Slot* slots, uint32_t b)
{
  Sector v;
  unsigned long long m0, m1;
  asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];"
      : "=l"(v.key[0]), "=l"(m0), "=l"(v.key[1]), "=l"(m1)
      : "l"(slots + 2 * static_cast<uint64_t>(b)));
  v.cnt[0]   = static_cast<uint32_t>(m0);
  v.first[0] = static_cast<uint32_t>(m0 >> 32);
  v.cnt[1]   = static_cast<uint32_t>(m1);
  v.first[1] = static_cast<uint32_t>(m1 >> 32);
  return v;
}

__global__ void k_pjoin_clear(const PackedTable t)
{
  for (uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s <= t.cap;
       s += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    reinterpret_cast<uint4*>(t.slots)[s] = make_uint4(0xffffffffu, 0xffffffffu, 0u, 0u);
}

// Every build row's representative (kNoSlot: a row that matches nothing) and
// its rank among its key's rows.  A new key's slot is claimed by one 128-bit
// compare-and-swap that writes the key, the count 1 and the representative
// together; a row of a known key adds 1 to the count and reads the
// representative beside it, in one 64-bit add.  Each row so touches one
// sector twice (20M unique keys, a 512 MB table: with the key claimed by
// itself and the count and the row stored after it 2,057 us, the join by row
// indices 933 us, this 1,397 us).
template <int KM>
__global__ void k_pjoin_build(const __grid_constant__ KeyPlan kp, int64_t n, const PackedTable t,
                              uint32_t* __restrict__ rep_of, uint32_t* __restrict__ rank_of)
{
  bool repeated = false;  // stored once a thread: a store a repeated key, all to one address, would queue
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    uint64_t k;
    if (!row_key<KM>(kp, r, k)) {
      rep_of[r] = kNoSlot;
      continue;
    }
    if (k == kEmptyWord) {
      const uint32_t rank = atomicAdd(&t.slots[t.cap].cnt, 1u);
      rep_of[r]           = static_cast<uint32_t>(n);
      rank_of[r]          = rank;
      if (rank == 0) t.slots[t.cap].first = static_cast<uint32_t>(r);
      else repeated = true;
      continue;
    }
    uint64_t s = 2 * (fmix64(k) & (t.cap / 2 - 1));
    for (uint64_t p = 0; p < t.cap; ++p) {  // cap > n: an empty slot is always met
      const uint64_t a = reinterpret_cast<uint64_t>(&t.slots[s].key);
      uint64_t cur     = Global::ld_u64(a);
      if (cur == kEmptyWord) {
        uint64_t old;
        Global::cas128(a, kEmptyWord, 0, k, (static_cast<uint64_t>(r) << 32) | 1u, cur, old);
        if (cur == kEmptyWord) {
          rep_of[r]  = static_cast<uint32_t>(r);
          rank_of[r] = 0;
          break;
        }
      }
      if (cur == k) {
        // cnt (low half) and representative (high half)
        const unsigned long long old = atomicAdd(reinterpret_cast<unsigned long long*>(a + 8), 1ULL);
        rep_of[r]                    = static_cast<uint32_t>(old >> 32);
        rank_of[r]                   = static_cast<uint32_t>(old);
        repeated                     = true;
        break;
      }
      s = (s + 1) & (t.cap - 1);
    }
  }
  if (repeated) *t.dup = 1u;
}

// With repeated keys: each key's row count at its representative (whose
// exclusive scan places the keys' runs in `rows`), read off the slots: adding
// the rows up again would queue on a key with many (1M rows of 100 keys 100 us).
__global__ void k_pjoin_counts(const PackedTable t, int64_t n, uint32_t* __restrict__ cnt)
{
  for (uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s <= t.cap;
       s += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(t.slots) + s);
    if (v.z != 0) cnt[s < t.cap ? v.w : static_cast<uint32_t>(n)] = v.z;
  }
}

// The build rows of each key next to each other, from start_of[representative].
__global__ void k_pjoin_place(int64_t n, const uint32_t* __restrict__ rep_of, const uint32_t* __restrict__ rank_of,
                              const uint32_t* __restrict__ start_of, int32_t* __restrict__ rows)
{
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const uint32_t k = rep_of[r];
    if (k != kNoSlot) rows[start_of[k] + rank_of[r]] = static_cast<int32_t>(r);
  }
}

// Output rows of a probe row whose key has `c` build rows.
__device__ __forceinline__ uint32_t rows_out(uint32_t c, int32_t kind)
{
  switch (kind) {
    case GBX_JOIN_INNER: return c;
    case GBX_JOIN_LEFT_SEMI: return c > 0 ? 1u : 0u;
    case GBX_JOIN_LEFT_ANTI: return c > 0 ? 0u : 1u;
    default: return c > 0 ? c : 1u;  // left, full
  }
}

__device__ __forceinline__ unsigned long long block_sum(unsigned long long v, unsigned long long* part)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long all = 0;
#pragma unroll
  for (int w = 0; w < kJBlock / 32; ++w) all += part[w];
  return all;
}

// match[r]: the matched build row (unique build keys) or slot (some key
// repeats), kNoSlot without a match; tile_out[tile]: the tile's output rows.
template <int KM>
__global__ void __launch_bounds__(kJBlock) k_pjoin_probe(const __grid_constant__ KeyPlan kp, int64_t n,
                                                         const PackedTable t, int32_t kind,
                                                         uint32_t* __restrict__ match,
                                                         int64_t* __restrict__ tile_out)
{
  __shared__ unsigned long long part[kJBlock / 32];
  const int64_t t0          = static_cast<int64_t>(blockIdx.x) * kJTile + threadIdx.x;
  const uint32_t mask       = static_cast<uint32_t>(t.cap / 2 - 1);
  const bool dup            = *t.dup != 0;
  const uint32_t all_ones   = t.slots[t.cap].cnt;  // the reserved slot: the all-ones key
  unsigned long long mine   = 0;
#pragma unroll 1
  for (int q0 = 0; q0 < kJPer; q0 += kJFlight) {
    const int64_t base = t0 + q0 * kJBlock;
    uint64_t k[kJFlight];
    uint32_t pending = 0;  // rows still probing
    uint32_t cnt[kJFlight], found[kJFlight], b[kJFlight];
#pragma unroll
    for (int q = 0; q < kJFlight; ++q) {
      const int64_t r = base + q * kJBlock;
      cnt[q]          = 0;
      found[q]        = kNoSlot;
      if (r < n && row_key<KM>(kp, r, k[q])) pending |= 1u << q;
    }
    Sector v[kJFlight];
#pragma unroll
    for (int q = 0; q < kJFlight; ++q) {
      if (!((pending >> q) & 1u)) continue;
      b[q] = static_cast<uint32_t>(fmix64(k[q])) & mask;
      v[q] = load_sector(t.slots, b[q]);
    }
    // every row still probing takes its next sector in the same round, so the
    // loads of a round overlap
    for (uint64_t p = 0; p <= mask && pending != 0; ++p) {
#pragma unroll
      for (int q = 0; q < kJFlight; ++q) {
        if (!((pending >> q) & 1u)) continue;
        const bool hi = v[q].key[1] == k[q];
        if (k[q] == kEmptyWord) {
          cnt[q] = all_ones;
          if (all_ones != 0) found[q] = dup ? static_cast<uint32_t>(t.cap) : t.slots[t.cap].first;
          pending &= ~(1u << q);
        } else if (hi || v[q].key[0] == k[q]) {
          cnt[q]   = hi ? v[q].cnt[1] : v[q].cnt[0];
          found[q] = dup ? 2 * b[q] + (hi ? 1u : 0u) : (hi ? v[q].first[1] : v[q].first[0]);
          pending &= ~(1u << q);
        } else if (v[q].key[0] == kEmptyWord || v[q].key[1] == kEmptyWord) {
          pending &= ~(1u << q);
        } else {
          b[q] = (b[q] + 1) & mask;
          v[q] = load_sector(t.slots, b[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kJFlight; ++q) {
      const int64_t r = base + q * kJBlock;
      if (r >= n) continue;
      match[r] = found[q];
      mine += rows_out(cnt[q], kind);
    }
  }
  const unsigned long long all = block_sum(mine, part);
  if (threadIdx.x == 0) tile_out[blockIdx.x] = static_cast<int64_t>(all);
}

// Output pairs when every probe row has at most one (unique build keys, or a
// semi / anti join), in probe-row order: a tile's matches are compacted
// through ballots, so a warp writes one contiguous run per load.
__global__ void __launch_bounds__(kJBlock) k_pjoin_emit_one(const uint32_t* __restrict__ match, int64_t n,
                                                            const int64_t* __restrict__ tile_at, int32_t kind,
                                                            int32_t* __restrict__ out_probe,
                                                            int32_t* __restrict__ out_build,
                                                            uint8_t* __restrict__ matched)
{
  __shared__ uint32_t cnt[kJPer][kJBlock / 32];
  const int lane   = threadIdx.x & 31;
  const int warp   = threadIdx.x >> 5;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * kJTile + threadIdx.x;
  uint32_t m[kJPer], bal[kJPer];
#pragma unroll
  for (int q = 0; q < kJPer; ++q) {
    const int64_t r = t0 + q * kJBlock;
    m[q]            = r < n ? __ldg(match + r) : kNoSlot;
  }
#pragma unroll
  for (int q = 0; q < kJPer; ++q) {
    const int64_t r = t0 + q * kJBlock;
    const bool has  = r < n && rows_out(m[q] != kNoSlot ? 1u : 0u, kind) != 0;
    bal[q]          = __ballot_sync(0xffffffffu, has);
    if (lane == 0) cnt[q][warp] = __popc(bal[q]);
  }
  __syncthreads();
  static_assert(kJPer * (kJBlock / 32) == 64, "two counts a lane of warp 0");
  if (warp == 0) {
    uint32_t* c      = &cnt[0][0];
    const uint32_t a = c[2 * lane], b = c[2 * lane + 1];
    uint32_t incl    = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    c[2 * lane]     = incl - a - b;
    c[2 * lane + 1] = incl - b;
  }
  __syncthreads();
  const int64_t base = tile_at[blockIdx.x];
  const bool pairs   = kind != GBX_JOIN_LEFT_SEMI && kind != GBX_JOIN_LEFT_ANTI;
#pragma unroll
  for (int q = 0; q < kJPer; ++q) {
    if (!((bal[q] >> lane) & 1u)) continue;
    const int64_t at = base + cnt[q][warp] + __popc(bal[q] & ((1u << lane) - 1u));
    out_probe[at]    = static_cast<int32_t>(t0 + q * kJBlock);
    if (!pairs) continue;
    out_build[at] = m[q] == kNoSlot ? kJoinNoneValue : static_cast<int32_t>(m[q]);
    if (matched != nullptr && m[q] != kNoSlot) matched[m[q]] = 1;
  }
}

// Output pairs when some build key repeats, in probe-row order.  A tile's
// outputs are shared among gridDim.y blocks, whatever the rows they come from:
// each block scans the tile's row counts and its threads look their outputs'
// rows up in the scan (a search of 11 steps in shared memory), so a warp writes
// 32 consecutive pairs.  Bound by the output's bytes where keys repeat often.
// Measured on B200 against one thread writing the runs of its probe rows one
// after another (8 rows a thread; 1 row a thread in the join by row indices):
// 10M probe rows of 4 pairs each 636 us (342), 100K of 1,000 2,646 us (1,916),
// 2,000 of 10,000 24,756 us (3,217); here 182, 353 and 97 us.
__global__ void __launch_bounds__(kJBlock) k_pjoin_emit_runs(const PackedTable t, int64_t nb,
                                                             const uint32_t* __restrict__ match,
                                                             int64_t n, const int64_t* __restrict__ tile_at,
                                                             int32_t kind, const uint32_t* __restrict__ start_of,
                                                             const int32_t* __restrict__ rows,
                                                             int32_t* __restrict__ out_probe,
                                                             int32_t* __restrict__ out_build,
                                                             uint8_t* __restrict__ matched)
{
  __shared__ __align__(16) uint32_t start[kJTile];  // a row's outputs, then its first output in the tile
  __shared__ uint32_t first[kJTile];                // its key's first position in `rows` (kNoSlot: none)
  __shared__ uint32_t part[kJBlock / 32];
  static_assert(kJPer == 8, "a thread scans two 16-byte vectors of counts");
  const int lane   = threadIdx.x & 31;
  const int warp   = threadIdx.x >> 5;
  const int64_t r0 = static_cast<int64_t>(blockIdx.x) * kJTile;
#pragma unroll
  for (int q = 0; q < kJPer; ++q) {
    const int i      = threadIdx.x + q * kJBlock;
    const uint32_t m = r0 + i < n ? __ldg(match + r0 + i) : kNoSlot;
    uint32_t cnt     = 0;
    first[i]         = kNoSlot;
    if (m != kNoSlot) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(t.slots) + m);
      cnt           = v.z;
      // (the reserved slot's representative is not in it)
      const uint32_t rep = m == t.cap ? static_cast<uint32_t>(nb) : v.w;
      first[i]           = __ldg(start_of + rep);
      if (matched != nullptr && blockIdx.y == 0) matched[rep] = 1;
    }
    start[i] = r0 + i < n ? rows_out(cnt, kind) : 0u;
  }
  __syncthreads();
  uint4* c         = reinterpret_cast<uint4*>(start) + threadIdx.x * 2;
  const uint4 c0   = c[0], c1 = c[1];
  const uint32_t s = c0.x + c0.y + c0.z + c0.w + c1.x + c1.y + c1.z + c1.w;  // a tile's outputs fit 31 bits
  uint32_t incl    = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) part[warp] = incl;
  __syncthreads();
  uint32_t at = incl - s, total = 0;
#pragma unroll
  for (int w = 0; w < kJBlock / 32; ++w) {
    if (w < warp) at += part[w];
    total += part[w];
  }
  uint4 f;
  f.x  = at;
  f.y  = f.x + c0.x;
  f.z  = f.y + c0.y;
  f.w  = f.z + c0.z;
  c[0] = f;
  f.x  = f.w + c0.w;
  f.y  = f.x + c1.x;
  f.z  = f.y + c1.y;
  f.w  = f.z + c1.z;
  c[1] = f;
  __syncthreads();
  const int64_t base = tile_at[blockIdx.x];
  const uint64_t lo  = static_cast<uint64_t>(total) * blockIdx.y / gridDim.y;
  const uint64_t hi  = static_cast<uint64_t>(total) * (blockIdx.y + 1) / gridDim.y;
  for (uint64_t o = lo + threadIdx.x; o < hi; o += kJBlock) {
    // the last row whose outputs begin at or before o (rows without outputs
    // begin where the next row does)
    uint32_t i = 0;
#pragma unroll
    for (uint32_t step = kJTile / 2; step > 0; step >>= 1)
      if (start[i + step] <= o) i += step;
    const uint32_t p  = first[i];
    out_probe[base + o] = static_cast<int32_t>(r0 + i);
    out_build[base + o] = p == kNoSlot ? kJoinNoneValue : rows[p + (static_cast<uint32_t>(o) - start[i])];
  }
}

// Full join: build rows whose key no probe row matched (`matched` is indexed
// by build row when keys are unique, else by the key's representative).
__global__ void k_pjoin_unmatched(const uint32_t* __restrict__ rep_of, int64_t n, bool repeated,
                                  const uint8_t* __restrict__ matched, uint32_t* __restrict__ flag)
{
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x)
    flag[r] = (rep_of[r] == kNoSlot || matched[repeated ? rep_of[r] : static_cast<uint32_t>(r)] == 0) ? 1u : 0u;
}

__global__ void k_pjoin_append(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ pos, int64_t n,
                               uint64_t base, int32_t* __restrict__ out_probe, int32_t* __restrict__ out_build)
{
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n;
       r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (!flag[r]) continue;
    out_probe[base + pos[r]] = kJoinNoneValue;
    out_build[base + pos[r]] = static_cast<int32_t>(r);
  }
}

int grid_for(int64_t n, int num_sms)
{
  const int64_t b = (n + kJBlock - 1) / kJBlock;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(b, int64_t(num_sms) * 8)));
}

// 1 / 2 when the key is one plain 8- / 4-byte column whose bits are the
// packed word, else 0.
int key_mode(const KeyPlan& kp)
{
  const KeyCol& kc = kp.cols[0];
  if (kp.ncols != 1 || kc.mask != nullptr || kc.is_float || kc.is_bool || kc.null_bit || kc.shift != 0) return 0;
  return kc.width == 8 ? 1 : kc.width == 4 ? 2 : 0;
}

// The sides' key plans with one layout: a column nullable on either side is
// nullable in both.  False when the key does not pack into one word.
bool join_key_plans(const gbx_table_view* build, const gbx_table_view* probe, int32_t compare_nulls, KeyPlan& kb,
                    KeyPlan& kp)
{
  const int ncols = build->num_columns;
  if (ncols > kMaxKeyCols) return false;
  std::vector<int64_t> nulls(ncols, 0);
  int bits = 0;
  for (int c = 0; c < ncols; ++c) {
    const gbx_column_view& b = build->columns[c];
    if (!is_fixed_width(b.type_id)) return false;
    bits += 8 * type_width(b.type_id);
    if (exact_null_count_or_neg(b) != 0 || exact_null_count_or_neg(probe->columns[c]) != 0) nulls[c] = -1;
  }
  if (bits > 64) return false;
  const int32_t policy = compare_nulls == GBX_NULLS_UNEQUAL ? GBX_NULL_EXCLUDE : GBX_NULL_INCLUDE;
  bool ok              = true;
  kb                   = make_key_plan(build->columns, ncols, policy, nulls, ok);
  if (!ok || kb.nwords != 1) return false;
  kp = make_key_plan(probe->columns, ncols, policy, nulls, ok);
  for (int c = 0; c < ncols; ++c) {
    // a side known to hold no nulls reads no mask
    if (exact_null_count_or_neg(build->columns[c]) == 0) kb.cols[c].mask = nullptr;
    if (exact_null_count_or_neg(probe->columns[c]) == 0) kp.cols[c].mask = nullptr;
  }
  return ok && kp.nwords == 1;
}

// Whether the packed table is the better one.  Its 16-byte slots are four times
// the bytes that the join by row indices probes, so once they leave L2 its
// build is the dearer one, and few probe rows do not earn that back.  Measured
// on B200, whole left joins, packed / by row indices, us (unique keys; keys
// drawn from as many as there are build rows):
//   5M build rows (134 MB), probe rows 1,000    323 / 380    379 / 365
//                                      nb / 8   338 / 431    407 / 425
//   20M build rows (537 MB),           1,000  1,595 / 1,316  1,724 / 1,631
//                                      nb / 8 1,688 / 1,572  1,869 / 1,848
//                                      nb / 4 1,781 / 1,823  1,988 / 2,053
//                                      nb     2,253 / 3,247  2,794 / 3,213
//   50M build rows (1.07 GB, load 0.74),   nb / 2 7,597 / 7,132
//                                          nb     9,087 / 10,210
bool packed_pays(int64_t nb, int64_t np, uint64_t cap, size_t l2_bytes)
{
  const size_t bytes = cap * sizeof(Slot);
  if (bytes <= l2_bytes) return true;
  if (bytes <= 2 * l2_bytes) return 16 * np >= nb;
  const bool loaded = 3 * static_cast<uint64_t>(nb) > 2 * cap;  // long probes
  return bytes > 6 * l2_bytes && loaded ? 4 * np >= 3 * nb : 4 * np > nb;
}

}  // namespace

bool packed_join(const gbx_table_view* build, const gbx_table_view* probe, int32_t compare_nulls, int32_t kind,
                 Alloc& a, gbx_column& out_probe, gbx_column& out_build)
{
  const int64_t nb = build->columns[0].size;
  const int64_t np = probe->columns[0].size;
  KeyPlan kb{}, kp{};
  if (nb == 0 || np == 0 || nb > kMaxBuildRows || !join_key_plans(build, probe, compare_nulls, kb, kp)) return false;
  cudaStream_t s       = a.st;
  const DeviceInfo dev = current_device();
  const int num_sms    = dev.num_sms;
  // load 0.375 to 0.75: at 1M build rows 32 MB of 16-byte slots, which stay
  // in L2 (a table twice that size does not fit beside the probe's streams)
  const uint64_t cap   = next_pow2(std::max<uint64_t>(static_cast<uint64_t>(nb) * 4 / 3 + 2, 64));
  if (!packed_pays(nb, np, cap, dev.l2_bytes)) return false;
  const int64_t ntiles = (np + kJTile - 1) / kJTile;

  Scratch sc(&a);
  const size_t nb4 = static_cast<size_t>(nb) * 4;
  PackedTable t{};
  t.cap         = cap;
  const size_t slot_bytes = (cap + 1) * sizeof(Slot) + kSectorBytes - 1;
  const size_t np4        = static_cast<size_t>(np) * 4;
  const size_t tile_bytes = static_cast<size_t>(ntiles + 1) * 8;
  size_t tb32 = 0, tb64 = 0;
  GBX_CUDA(scan_exclusive_u32(nullptr, nullptr, nb + 1, nullptr, &tb32, s));
  GBX_CUDA(scan_exclusive_i64(nullptr, nullptr, ntiles + 1, nullptr, &tb64, s));
  size_t tbytes = std::max(std::max(tb32, tb64), size_t(1));
  sc.together({slot_bytes, 8, nb4, nb4, np4, tile_bytes, tbytes});
  // 32-byte sectors, whatever the caller's allocator aligns to
  const auto raw = reinterpret_cast<uintptr_t>(sc.get(slot_bytes));
  t.slots        = reinterpret_cast<Slot*>((raw + kSectorBytes - 1) & ~(kSectorBytes - 1));
  t.dup         = static_cast<uint32_t*>(sc.get(8));
  auto* rep_of  = static_cast<uint32_t*>(sc.get(nb4));
  auto* rank_of = static_cast<uint32_t*>(sc.get(nb4));
  auto* match   = static_cast<uint32_t*>(sc.get(np4));
  auto* tiles   = static_cast<int64_t*>(sc.get(tile_bytes));
  void* temp    = sc.get(tbytes);

  // 1. the table
  GBX_CUDA(cudaMemsetAsync(t.dup, 0, 8, s));
  k_pjoin_clear<<<grid_for(static_cast<int64_t>(cap) + 1, num_sms), kJBlock, 0, s>>>(t);
  const int gb = grid_for(nb, num_sms);
  switch (key_mode(kb)) {
    case 1: k_pjoin_build<1><<<gb, kJBlock, 0, s>>>(kb, nb, t, rep_of, rank_of); break;
    case 2: k_pjoin_build<2><<<gb, kJBlock, 0, s>>>(kb, nb, t, rep_of, rank_of); break;
    default: k_pjoin_build<0><<<gb, kJBlock, 0, s>>>(kb, nb, t, rep_of, rank_of); break;
  }
  GBX_CUDA(cudaGetLastError());

  // 2. matches and output rows per tile
  const int gp = static_cast<int>(ntiles);
  switch (key_mode(kp)) {
    case 1: k_pjoin_probe<1><<<gp, kJBlock, 0, s>>>(kp, np, t, kind, match, tiles); break;
    case 2: k_pjoin_probe<2><<<gp, kJBlock, 0, s>>>(kp, np, t, kind, match, tiles); break;
    default: k_pjoin_probe<0><<<gp, kJBlock, 0, s>>>(kp, np, t, kind, match, tiles); break;
  }
  GBX_CUDA(cudaGetLastError());
  GBX_CUDA(cudaMemsetAsync(tiles + ntiles, 0, 8, s));
  GBX_CUDA(scan_exclusive_i64(tiles, tiles, ntiles + 1, temp, &tbytes, s));
  int64_t total  = 0;
  uint32_t h_dup = 0;
  GBX_CUDA(cudaMemcpyAsync(&total, tiles + ntiles, 8, cudaMemcpyDeviceToHost, s));
  GBX_CUDA(cudaMemcpyAsync(&h_dup, t.dup, 4, cudaMemcpyDeviceToHost, s));
  GBX_CUDA(cudaStreamSynchronize(s));
  GBX_EXPECTS(total <= INT32_MAX, "the join's output exceeds cudf::size_type rows");

  // 3. outputs (a full join's size is known once the matches are marked)
  const bool full  = kind == GBX_JOIN_FULL;
  const bool pairs = kind != GBX_JOIN_LEFT_SEMI && kind != GBX_JOIN_LEFT_ANTI;
  const bool one   = h_dup == 0 || !pairs;
  uint8_t* matched = nullptr;
  uint32_t* start_of = nullptr;
  int32_t* rows      = nullptr;
  if (!one) {
    // each key's rows next to each other (entry nb: the all-ones key)
    sc.together({nb4 + 4, nb4 + 4, nb4});
    auto* cnt = static_cast<uint32_t*>(sc.get(nb4 + 4));
    start_of  = static_cast<uint32_t*>(sc.get(nb4 + 4));
    rows      = static_cast<int32_t*>(sc.get(nb4));
    GBX_CUDA(cudaMemsetAsync(cnt, 0, nb4 + 4, s));
    k_pjoin_counts<<<grid_for(static_cast<int64_t>(cap) + 1, num_sms), kJBlock, 0, s>>>(t, nb, cnt);
    GBX_CUDA(cudaGetLastError());
    GBX_CUDA(scan_exclusive_u32(cnt, start_of, nb + 1, temp, &tbytes, s));
    k_pjoin_place<<<gb, kJBlock, 0, s>>>(nb, rep_of, rank_of, start_of, rows);
    GBX_CUDA(cudaGetLastError());
  }
  int32_t *probe_buf = nullptr, *build_buf = nullptr;
  if (full) {
    matched = static_cast<uint8_t*>(sc.get(static_cast<size_t>(nb) + 1));
    GBX_CUDA(cudaMemsetAsync(matched, 0, static_cast<size_t>(nb) + 1, s));
    probe_buf = static_cast<int32_t*>(sc.get(static_cast<size_t>(total) * 4));
    build_buf = static_cast<int32_t*>(sc.get(static_cast<size_t>(total) * 4));
  } else {
    alloc_column(a, out_probe, GBX_TYPE_INT32, 0, total, false);
    alloc_column(a, out_build, GBX_TYPE_INT32, 0, pairs ? total : 0, false);
    probe_buf = static_cast<int32_t*>(out_probe.data);
    build_buf = static_cast<int32_t*>(out_build.data);
  }
  if (total > 0) {
    if (one) k_pjoin_emit_one<<<gp, kJBlock, 0, s>>>(match, np, tiles, kind, probe_buf, build_buf, matched);
    else {
      // blocks a tile: one per kEmitPart outputs of the average tile, more
      // where that leaves SMs idle
      const int64_t tile_out = total / ntiles;
      const int64_t idle     = std::min<int64_t>((2 * num_sms + ntiles - 1) / ntiles, tile_out / kEmitLeast);
      const int64_t parts    = std::max<int64_t>(1, std::min<int64_t>(std::max(tile_out / kEmitPart, idle), 65535));
      k_pjoin_emit_runs<<<dim3(gp, static_cast<unsigned>(parts)), kJBlock, 0, s>>>(
        t, nb, match, np, tiles, kind, start_of, rows, probe_buf, build_buf, matched);
    }
    GBX_CUDA(cudaGetLastError());
  }
  if (full) {
    auto* flag = static_cast<uint32_t*>(sc.get(nb4));
    auto* pos  = static_cast<uint32_t*>(sc.get(nb4));
    k_pjoin_unmatched<<<gb, kJBlock, 0, s>>>(rep_of, nb, !one, matched, flag);
    GBX_CUDA(cudaGetLastError());
    GBX_CUDA(scan_exclusive_u32(flag, pos, nb, temp, &tbytes, s));
    uint32_t last[2] = {0, 0};
    GBX_CUDA(cudaMemcpyAsync(&last[0], pos + nb - 1, 4, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaMemcpyAsync(&last[1], flag + nb - 1, 4, cudaMemcpyDeviceToHost, s));
    GBX_CUDA(cudaStreamSynchronize(s));
    const int64_t unmatched = static_cast<int64_t>(last[0]) + last[1];
    const int64_t m         = total + unmatched;
    alloc_column(a, out_probe, GBX_TYPE_INT32, 0, m, false);
    alloc_column(a, out_build, GBX_TYPE_INT32, 0, m, false);
    if (total > 0) {
      GBX_CUDA(cudaMemcpyAsync(out_probe.data, probe_buf, total * 4, cudaMemcpyDeviceToDevice, s));
      GBX_CUDA(cudaMemcpyAsync(out_build.data, build_buf, total * 4, cudaMemcpyDeviceToDevice, s));
    }
    if (unmatched > 0) {
      k_pjoin_append<<<gb, kJBlock, 0, s>>>(flag, pos, nb, static_cast<uint64_t>(total),
                                            static_cast<int32_t*>(out_probe.data),
                                            static_cast<int32_t*>(out_build.data));
      GBX_CUDA(cudaGetLastError());
    }
  }
  GBX_CUDA(cudaStreamSynchronize(s));
  return true;
}

}  // namespace gbx
