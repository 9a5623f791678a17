// gbx_tiled.cu -- aggregation by grouping each tile of rows in shared memory
// before touching the CTA's table.
//
// Applying rows one by one to a shared table costs ~13 shared-memory atomics
// a row for the 100M-row workload's 12 accumulators, and the 64-bit ones run
// as compare-and-swap loops that conflict when many lanes hit the same few
// slots (35.7 warp-instructions a row).  Here a CTA takes up to 8 rows a
// thread at a time and
//   1. packs the tile's keys column by column (one uniform branch on a key
//      column's width serves all of a thread's rows), finds each row's slot
//      in its table and takes the next rank of that slot with one 32-bit
//      shared atomic; rows whose key finds no slot are listed and sent to the
//      global table by the whole CTA together;
//   2. scans the slots' (rows, chunks of at most kChunk rows) in one pass;
//   3. stores each channel's values, at their own width, at their row's
//      position, so that the tile lies in shared memory group by group (the
//      first channel's loads are in flight across the scan);
//   4. folds one chunk per thread in registers, four consecutive values at a
//      time, and merges it into the group's slot with shared atomics; a warp
//      whose 32 chunks are all of one group adds them with shuffles first.
// After its last tile the CTA merges its table into the global one, as the
// reference's shared-memory aggregation does (hash/groupby.cu:424-504).
//
// Issue-bound (57% of issue slots, 16.6 warp-instructions a row): the work per
// row is a hash, a probe, a rank, one staged store and load per channel and
// the fold itself.  The warp meets again after every probe loop and every
// compare-and-swap loop; where it did not, the lanes ran all that followed
// apart (11 active lanes an instruction, 33 warp-instructions a row).  The four-wide folds keep the
// tests for the accumulators a plan uses, and the loop control, at a quarter
// of an instruction a row.  Two CTAs of 512 threads an SM where the table and
// the tile fit half its shared memory, so that one folds while the other
// waits for its loads; one of 1,024 threads for larger tables.
//
// The caller's rows are dealt to the CTAs tile by tile; the bucket-ordered
// copies of the radix partitioning (PART) in one contiguous run per CTA.
//
// Measured on B200, 100M rows, 12 accumulators, against the kernel this
// replaces (per-slot folds of values read through a permutation, the warp
// apart after each probe): 100 groups 3,586 -> 2,528 us, bucket-ordered copies
// of 1e4 groups 4,257 -> 2,608 us; 10M rows, 1,000 groups, five aggregations
// of one double column, 384 us with per-row shared atomics -> 254 us.
#include <algorithm>
#include <type_traits>

#include "gbx_rows.cuh"
#include "gbx_warpcore.cuh"

namespace gbx {

using namespace dev;

namespace {

constexpr int kPer           = 8;  // rows per thread and tile at most
constexpr int kBatch         = 4;  // of which so many are in flight together
constexpr int kChunk         = 16; // rows of one group folded by one thread
constexpr int kMaxSlots      = 4096;
constexpr uint32_t kNoRec    = 0xffffffffu;
// dynamic shared memory so that two CTAs of 512 threads fit an SM (228 KB,
// less 1 KB reserved and the static shared memory per CTA), or one of 1,024
constexpr size_t kSmemTwo = 112 * 1024;
constexpr size_t kSmemOne = 225 * 1024;

// Byte offsets of the per-tile areas in dynamic shared memory, after the
// table: slot counts ((S + 1) u32), each slot's first position and chunk
// ((S + 2) u32: chunk << 16 | position), each row's slot and rank (u32), the
// slot of each chunk (u16), the rows that found no slot (u16), each channel's values at their width, and a
// validity byte per row of a nullable channel.
struct TiledLayout {
  uint32_t cnt_off, oc_off, rec_off, cslot_off, spill_off, total;
  uint32_t val_off[kMaxChannels];
  uint32_t ok_off[kMaxChannels];  // 0: the channel has no nulls
  int tile_rows;
  int block;
};

TiledLayout tiled_layout(const SmemLayout& sl, const Plan& p, int block, int tile_rows)
{
  TiledLayout tl{};
  tl.block     = block;
  tl.tile_rows = tile_rows;
  uint32_t o   = (sl.total + 15) & ~15u;
  tl.cnt_off   = o;
  o += (sl.slots + 1) * 4;
  tl.oc_off = o;
  o += (sl.slots + 2) * 4;
  tl.rec_off = o;
  o += tile_rows * 4;
  tl.cslot_off = o;
  o += (tile_rows / kChunk + sl.slots + 2) * 2;
  tl.spill_off = o;
  o += tile_rows * 2;
  for (int c = 0; c < p.nchan; ++c) {
    o             = (o + 15) & ~15u;
    tl.val_off[c] = o;
    o += tile_rows * pt_width(p.chan[c].ptype);
    if (p.chan[c].a_cnt >= 0) {
      tl.ok_off[c] = o;
      o += tile_rows;
    }
  }
  tl.total = (o + 15) & ~15u;
  return tl;
}

// The largest tile that fits: two CTAs an SM when at least half a full tile
// does, else one; tile_rows 0 when none fits.
TiledLayout pick_tiled_layout(const SmemLayout& sl, const Plan& p)
{
  for (int rows = 512 * kPer; rows >= 512 * (kPer / 2); rows -= 512) {
    const TiledLayout tl = tiled_layout(sl, p, 512, rows);
    if (tl.total <= kSmemTwo) return tl;
  }
  for (int rows = 1024 * kPer; rows >= 1024; rows -= 1024) {
    const TiledLayout tl = tiled_layout(sl, p, 1024, rows);
    if (tl.total <= kSmemOne) return tl;
  }
  return TiledLayout{};
}

// Channel c's value bits and validity (bit q of the result) of this thread's
// rows r0 + q * step (a plain or copied column).
template <bool PART>
__device__ __forceinline__ uint32_t channel_rows(const Plan& plan, const PartBufs& pb, int c, int64_t r0, int step,
                                                 uint32_t rows, uint64_t (&v)[kBatch])
{
  if constexpr (PART) {
    const PartCol& pc = pb.col[c];
    load_rows<kBatch>(pc.width, pc.vals, r0, step, rows, v);
    uint32_t ok = rows;
    if (pc.valid != nullptr) {
#pragma unroll
      for (int q = 0; q < kBatch; ++q)
        if (((rows >> q) & 1u) && __ldg(pc.valid + r0 + static_cast<int64_t>(q) * step) == 0) ok &= ~(1u << q);
    }
    return ok;
  } else {
    const Channel& ch = plan.chan[c];
    load_rows<kBatch>(pt_width(ch.ptype), ch.data, r0 + ch.offset, step, rows, v);
    return valid_rows<kBatch>(ch.mask, r0 + ch.offset, step, rows);
  }
}

// The same through a dictionary, for the rows that found a slot only (an
// excluded row's index is not looked at).
__device__ __noinline__ uint32_t dict_rows(const Plan& plan, int c, int64_t r0, int step, uint32_t rows,
                                           uint64_t (&v)[kBatch], int32_t* status)
{
  const RowSource src{&plan};
  uint32_t ok = 0;
  for (int q = 0; q < kBatch; ++q) {
    v[q] = 0;
    if (((rows >> q) & 1u) && src.value(c, r0 + static_cast<int64_t>(q) * step, v[q], status)) ok |= 1u << q;
  }
  return ok;
}

// ------------------------------------------------------------- the fold

template <int PT>
struct Staged {
  using type = unsigned long long;
};
template <>
struct Staged<P_I8> { using type = uint8_t; };
template <>
struct Staged<P_U8> { using type = uint8_t; };
template <>
struct Staged<P_BOOL> { using type = uint8_t; };
template <>
struct Staged<P_I16> { using type = uint16_t; };
template <>
struct Staged<P_U16> { using type = uint16_t; };
template <>
struct Staged<P_I32> { using type = uint32_t; };
template <>
struct Staged<P_U32> { using type = uint32_t; };
template <>
struct Staged<P_F32> { using type = uint32_t; };

// 64-bit integer add to a shared word as two 32-bit ones (the carry follows
// from the low half's old value): the 32-bit adds are native, a 64-bit one is
// a compare-and-swap loop.
__device__ __forceinline__ void shared_add_i64(uint64_t* p, uint64_t x)
{
  uint32_t* w        = reinterpret_cast<uint32_t*>(p);
  const uint32_t lo  = static_cast<uint32_t>(x);
  const uint32_t old = atomicAdd(w, lo);
  const uint32_t hi  = static_cast<uint32_t>(x >> 32) + (old + lo < old ? 1u : 0u);
  if (hi != 0) atomicAdd(w + 1, hi);
}

__device__ __forceinline__ uint64_t shfl_down_u64(uint64_t v, int o)
{
  return static_cast<uint64_t>(__shfl_down_sync(kFull, static_cast<unsigned long long>(v), o));
}

// Folds one chunk (staged positions p0 .. p0 + len) of a channel of physical
// type PT in registers and merges it into slot s of the CTA table at `smem`;
// `uniform`: the warp's 32 chunks are all of slot s (all 32 lanes call it).
// The VAR sums are relative to the slot's shift, which the first chunk with a
// valid non-NaN value records.  Nulls are folded as identities.
template <int PT>
__device__ __forceinline__ void fold_chunk(const Channel& ch, unsigned char* smem, const SmemLayout& sl,
                                           uint32_t val_off, uint32_t ok_off, uint32_t p0, uint32_t len, uint32_t s,
                                           bool uniform, uint32_t lanes, int32_t* status)
{
  constexpr bool kFloat = PT == P_F32 || PT == P_F64;
  constexpr bool kM64   = PT == P_I64 || PT == P_U64 || PT == P_F64;
  using T               = typename Staged<PT>::type;
  using M               = typename std::conditional<kM64, uint64_t, uint32_t>::type;
  const T* vals         = reinterpret_cast<const T*>(smem + val_off) + p0;
  const uint8_t* oks    = ok_off ? smem + ok_off + p0 : nullptr;
  const uint32_t roles  = chan_roles(ch);

  uint32_t cnt = 0;
  M mn = static_cast<M>(~0ULL), mx = 0;
  uint64_t sum = 0, sq = 0, prod = 1;  // integer channels
  double fsum = 0.0, fsq = 0.0, fprod = 1.0, s2 = 0.0, s1 = 0.0, K = 0.0;
  if (roles & R_VAR) {
    uint64_t* kp = reinterpret_cast<uint64_t*>(smem + sl.acc_off[ch.a_k]) + s;
    uint64_t kb  = *kp;
    if (kb == kShiftUnset) {
      for (uint32_t j = 0; j < len; ++j) {
        if (oks != nullptr && !oks[j]) continue;
        const double x = as_f64(vals[j], PT);
        if (x != x) continue;
        const uint64_t xb = static_cast<uint64_t>(__double_as_longlong(x));
        kb = atomicCAS(reinterpret_cast<unsigned long long*>(kp), static_cast<unsigned long long>(kShiftUnset),
                       static_cast<unsigned long long>(xb));
        if (kb == kShiftUnset) kb = xb;
        break;
      }
    }
    K = __longlong_as_double(static_cast<long long>(kb));
    __syncwarp(lanes);
  }
  for (uint32_t j0 = 0; j0 < len; j0 += 4) {
    uint64_t b[4];
    bool ok[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t j = j0 + i;
      ok[i]            = j < len;
      b[i]             = ok[i] ? static_cast<uint64_t>(vals[j]) : 0;
      if (oks != nullptr) ok[i] = ok[i] && oks[j] != 0;
      cnt += ok[i] ? 1u : 0u;
    }
    if (roles & (R_MIN | R_MAX)) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (roles & R_MIN) mn = min(mn, ok[i] ? static_cast<M>(enc_minmax(b[i], PT, true)) : static_cast<M>(~0ULL));
        if (roles & R_MAX) mx = max(mx, ok[i] ? static_cast<M>(enc_minmax(b[i], PT, false)) : static_cast<M>(0));
      }
    }
    if constexpr (kFloat) {
      double x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = ok[i] ? as_f64(b[i], PT) : 0.0;
      if (roles & R_SUM) {
#pragma unroll
        for (int i = 0; i < 4; ++i) fsum += x[i];
      }
      if (roles & R_VAR) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double d = ok[i] ? x[i] - K : 0.0;
          s2 += d * d;
          s1 += d;
        }
      }
      if (roles & R_SQ) {
#pragma unroll
        for (int i = 0; i < 4; ++i) fsq += x[i] * x[i];
      }
      if (roles & R_PROD) {
#pragma unroll
        for (int i = 0; i < 4; ++i) fprod *= ok[i] ? x[i] : 1.0;
      }
    } else {
      int64_t x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = ok[i] ? as_i64(b[i], PT) : 0;
      if (roles & R_SUM) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sum += static_cast<uint64_t>(x[i]);
      }
      if (roles & R_VAR) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double xf = PT == P_U64 ? static_cast<double>(static_cast<uint64_t>(x[i])) : static_cast<double>(x[i]);
          const double d  = ok[i] ? xf - K : 0.0;
          s2 += d * d;
        }
      }
      if (roles & R_SQ) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sq += static_cast<uint64_t>(x[i]) * static_cast<uint64_t>(x[i]);
      }
      if (roles & R_PROD) {
#pragma unroll
        for (int i = 0; i < 4; ++i) prod *= ok[i] ? static_cast<uint64_t>(x[i]) : 1ULL;
      }
    }
  }
  __syncwarp(lanes);
  if (uniform) {
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
      cnt += __shfl_down_sync(kFull, cnt, o);
      if (roles & R_MIN) {
        if constexpr (kM64) mn = min(mn, static_cast<M>(shfl_down_u64(mn, o)));
        else mn = min(mn, static_cast<M>(__shfl_down_sync(kFull, mn, o)));
      }
      if (roles & R_MAX) {
        if constexpr (kM64) mx = max(mx, static_cast<M>(shfl_down_u64(mx, o)));
        else mx = max(mx, static_cast<M>(__shfl_down_sync(kFull, mx, o)));
      }
      if constexpr (kFloat) {
        if (roles & R_SUM) fsum += __shfl_down_sync(kFull, fsum, o);
        if (roles & R_SQ) fsq += __shfl_down_sync(kFull, fsq, o);
        if (roles & R_PROD) fprod *= __shfl_down_sync(kFull, fprod, o);
      } else {
        if (roles & R_SUM) sum += shfl_down_u64(sum, o);
        if (roles & R_SQ) sq += shfl_down_u64(sq, o);
        if (roles & R_PROD) prod *= shfl_down_u64(prod, o);
      }
      if (roles & R_VAR) {
        s2 += __shfl_down_sync(kFull, s2, o);
        s1 += __shfl_down_sync(kFull, s1, o);
      }
    }
  }
  // the lanes meet again after every compare-and-swap loop (floating adds), or
  // the rest of the merge and the next channel would run apart
  const bool mine = cnt != 0 && (!uniform || (threadIdx.x & 31) == 0);
  if (mine) {
    if (ch.a_cnt >= 0) atomicAdd(reinterpret_cast<uint32_t*>(smem + sl.acc_off[ch.a_cnt]) + s, cnt);
    // a slot's extremes settle early: most chunks only read them
    if (roles & R_MIN) {
      M* p = reinterpret_cast<M*>(smem + sl.acc_off[ch.a_min]) + s;
      if constexpr (kM64) {
        if (mn < *p) atomicMin(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(mn));
      } else {
        if (mn < *p) atomicMin(reinterpret_cast<uint32_t*>(p), static_cast<uint32_t>(mn));
      }
    }
    if (roles & R_MAX) {
      M* p = reinterpret_cast<M*>(smem + sl.acc_off[ch.a_max]) + s;
      if constexpr (kM64) {
        if (mx > *p) atomicMax(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(mx));
      } else {
        if (mx > *p) atomicMax(reinterpret_cast<uint32_t*>(p), static_cast<uint32_t>(mx));
      }
    }
    if constexpr (!kFloat) {
      if (roles & R_SUM) shared_add_i64(reinterpret_cast<uint64_t*>(smem + sl.acc_off[ch.a_sum]) + s, sum);
      if (roles & R_SQ) shared_add_i64(reinterpret_cast<uint64_t*>(smem + sl.acc_off[ch.a_sq]) + s, sq);
    }
  }
  __syncwarp(lanes);
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  if constexpr (kFloat) {
    if (roles & R_SUM) {
      if (mine) atomicAdd(reinterpret_cast<double*>(smem + sl.acc_off[ch.a_sum]) + s, fsum);
      __syncwarp(lanes);
    }
    if (roles & R_SQ) {
      if (mine) atomicAdd(reinterpret_cast<double*>(smem + sl.acc_off[ch.a_sq]) + s, fsq);
      __syncwarp(lanes);
    }
    if (roles & R_PROD) {
      if (mine) mul_cas_f64<Shared>(base + sl.acc_off[ch.a_prod] + s * 8, fprod, status);
      __syncwarp(lanes);
    }
    if (roles & R_VAR) {
      if (mine) atomicAdd(reinterpret_cast<double*>(smem + sl.acc_off[ch.a_s1]) + s, s1);
      __syncwarp(lanes);
    }
  } else if (roles & R_PROD) {
    if (mine) mul_cas_i64<Shared>(base + sl.acc_off[ch.a_prod] + s * 8, static_cast<int64_t>(prod), status);
    __syncwarp(lanes);
  }
  if (roles & R_VAR) {
    if (mine) atomicAdd(reinterpret_cast<double*>(smem + sl.acc_off[ch.a_s2]) + s, s2);
    __syncwarp(lanes);
  }
}

// The rows q0 .. q0 + kBatch - 1 of a thread that lie in its tile (`per` rows
// a thread) and below n, as bits; r0 is row q0.
__device__ __forceinline__ uint32_t in_tile(int q0, int per, int64_t r0, int step, int64_t n)
{
  uint32_t m = 0;
#pragma unroll
  for (int q = 0; q < kBatch; ++q)
    if (q0 + q < per && r0 + q * step < n) m |= 1u << q;
  return m;
}

// The listed rows of a tile: straight into the global table.
template <int NW, bool PART>
__device__ __noinline__ void spill_rows(const Plan& plan, const TableRef& t, const PartBufs& pb, const uint16_t* list,
                                        uint32_t n, int64_t t0, uint32_t max_probes)
{
  const Level<Global> G = global_level(t);
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const int64_t r = t0 + list[i];
    uint64_t k[NW];
    if constexpr (PART) PartSource{&pb}.key<NW>(r, k);
    else pack_key<NW>(plan.key, r, k);
    const int64_t g = global_slot<NW>(t, k, max_probes);
    if (g < 0) continue;
    if constexpr (PART) accumulate_row_from<Global>(plan, PartSource{&pb}, G, g, r, t.status);
    else accumulate_row<Global>(plan, G, g, r, t.status);
  }
}

template <int NW, bool PART, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) k_agg_tiled(const __grid_constant__ Plan plan,
                                                               const __grid_constant__ TableRef t,
                                                               const __grid_constant__ SmemLayout sl,
                                                               const __grid_constant__ TiledLayout tl, int64_t n,
                                                               const __grid_constant__ PartBufs pb,
                                                               const uint32_t* n_part, uint32_t smem_probes,
                                                               uint32_t max_probes)
{
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kWarps = BLOCK / 32;
  __shared__ uint32_t s_warp[kWarps];
  __shared__ uint32_t s_nspill;
  const uint32_t S    = sl.slots;
  const int tile_rows = tl.tile_rows;
  const int per       = tile_rows / BLOCK;
  const int lane      = threadIdx.x & 31;
  const int warp      = threadIdx.x >> 5;
  uint64_t* skeys     = reinterpret_cast<uint64_t*>(smem + sl.keys_off);
  uint32_t* srows     = reinterpret_cast<uint32_t*>(smem + sl.rows_off);
  uint32_t* cnt       = reinterpret_cast<uint32_t*>(smem + tl.cnt_off);
  uint32_t* oc        = reinterpret_cast<uint32_t*>(smem + tl.oc_off);
  uint32_t* rec       = reinterpret_cast<uint32_t*>(smem + tl.rec_off);
  uint16_t* cslot     = reinterpret_cast<uint16_t*>(smem + tl.cslot_off);
  uint16_t* spill     = reinterpret_cast<uint16_t*>(smem + tl.spill_off);
  const uint32_t keys_sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + sl.keys_off;

  // identity fill, counts zeroed
  for (uint32_t s = threadIdx.x; s <= S; s += BLOCK) {
#pragma unroll
    for (int w = 0; w < NW; ++w) skeys[s * NW + w] = kEmptyWord;
    srows[s] = 0;
    cnt[s]   = 0;
  }
  for (int a = 0; a < plan.acc.nacc; ++a) {
    const uint64_t id = identity_bits(plan.acc.kind[a]);
    if (acc_bytes(plan.acc.kind[a]) == 4) {
      uint32_t* p = reinterpret_cast<uint32_t*>(smem + sl.acc_off[a]);
      for (uint32_t s = threadIdx.x; s <= S; s += BLOCK) p[s] = static_cast<uint32_t>(id);
    } else {
      uint64_t* p = reinterpret_cast<uint64_t*>(smem + sl.acc_off[a]);
      for (uint32_t s = threadIdx.x; s <= S; s += BLOCK) p[s] = id;
    }
  }
  if (threadIdx.x == 0) s_nspill = 0;
  __syncthreads();

  if constexpr (PART) n = *n_part;
  const int64_t ntiles     = (n + tile_rows - 1) / tile_rows;
  const int64_t tile_begin = PART ? ntiles * blockIdx.x / gridDim.x : blockIdx.x;
  const int64_t tile_end   = PART ? ntiles * (blockIdx.x + 1) / gridDim.x : ntiles;
  const int64_t tile_step  = PART ? 1 : gridDim.x;
  const uint32_t slots_per = (S + 1 + BLOCK - 1) / BLOCK;  // slots scanned by one thread
  for (int64_t tile = tile_begin; tile < tile_end; tile += tile_step) {
    const int64_t t0 = tile * tile_rows;
    // 1. slot and rank of each row (kNoRec: no row, excluded, or listed)
#pragma unroll 1
    for (int q0 = 0; q0 < per; q0 += kBatch) {
      const int64_t r0 = t0 + threadIdx.x + q0 * BLOCK;
      uint32_t kept    = in_tile(q0, per, r0, BLOCK, n);
      uint64_t k[kBatch][NW];
      if constexpr (PART) {
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
#pragma unroll
          for (int w = 0; w < NW; ++w) k[q][w] = ((kept >> q) & 1u) ? __ldg(pb.keys[w] + r0 + q * BLOCK) : 0;
      } else {
        kept = pack_rows<kBatch, NW>(plan.key, PlanKeyBufs{&plan.key}, r0, BLOCK, kept, k);
      }
      uint32_t slot[kBatch];
      const uint32_t found = find_slots<kBatch, NW>(skeys, keys_sa, S - 1, kept, k, smem_probes, slot);
      if (__any_sync(kFull, found != kept)) {
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
          if (((kept & ~found) >> q) & 1u)
            spill[atomicAdd(&s_nspill, 1u)] = static_cast<uint16_t>(threadIdx.x + (q0 + q) * BLOCK);
        __syncwarp();
      }
#pragma unroll
      for (int q = 0; q < kBatch; ++q) {
        if (q0 + q >= per) break;
        rec[threadIdx.x + (q0 + q) * BLOCK] =
          ((found >> q) & 1u) ? (slot[q] << 16) | atomicAdd(cnt + slot[q], 1u) : kNoRec;
      }
    }
    // the first values load across the scan
    uint64_t v[kBatch];
    uint32_t ok = 0;
    if (plan.nchan > 0 && (PART || plan.chan[0].dict_data == nullptr)) {
      const int64_t r0 = t0 + threadIdx.x;
      ok               = channel_rows<PART>(plan, pb, 0, r0, BLOCK, in_tile(0, per, r0, BLOCK, n), v);
    }
    __syncthreads();
    const uint32_t nspill = s_nspill;
    // 2. (chunks << 16 | rows) scanned over the slots
    uint32_t sum = 0;
    for (uint32_t q = 0; q < slots_per; ++q) {
      const uint32_t s = threadIdx.x * slots_per + q;
      const uint32_t c = s <= S ? cnt[s] : 0u;
      sum += c | (((c + kChunk - 1) / kChunk) << 16);
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t total;
    {
      const uint32_t w = lane < kWarps ? s_warp[lane] : 0u;
      uint32_t wi      = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(kFull, wi, o);
        if (lane >= o) wi += x;
      }
      total        = __shfl_sync(kFull, wi, 31);
      uint32_t run = __shfl_sync(kFull, wi - w, warp) + incl - sum;
      for (uint32_t q = 0; q < slots_per; ++q) {
        const uint32_t s = threadIdx.x * slots_per + q;
        if (s > S) break;
        const uint32_t c  = cnt[s];
        const uint32_t nc = (c + kChunk - 1) / kChunk;
        oc[s]             = run;
        if (c != 0) {
          srows[s] += c;
          cnt[s] = 0;
          for (uint32_t j = 0; j < nc; ++j) cslot[(run >> 16) + j] = static_cast<uint16_t>(s);
        }
        run += c | (nc << 16);
      }
      if (threadIdx.x == 0) {
        oc[S + 1] = total;
        s_nspill  = 0;
      }
    }
    __syncthreads();
    // 3. the values, group by group; the next values load while these are
    //    stored
#pragma unroll 1
    for (int q0 = 0; q0 < per; q0 += kBatch) {
      const int64_t r0 = t0 + threadIdx.x + q0 * BLOCK;
      uint32_t pos[kBatch];
      uint32_t rows = 0;
#pragma unroll
      for (int q = 0; q < kBatch; ++q) {
        pos[q] = q0 + q < per ? rec[threadIdx.x + (q0 + q) * BLOCK] : kNoRec;
        if (pos[q] != kNoRec) {
          rows |= 1u << q;
          pos[q] = (oc[pos[q] >> 16] & 0xffffu) + (pos[q] & 0xffffu);
        }
      }
#pragma unroll 1
      for (int c = 0; c < plan.nchan; ++c) {
        if (!PART && plan.chan[c].dict_data != nullptr) ok = dict_rows(plan, c, r0, BLOCK, rows, v, t.status);
        uint64_t vn[kBatch] = {};
        uint32_t okn        = 0;
        {
          const bool last = c + 1 == plan.nchan;
          const int cn    = last ? 0 : c + 1;
          const int qn    = last ? q0 + kBatch : q0;
          if (qn < per && (PART || plan.chan[cn].dict_data == nullptr)) {
            const int64_t rn = t0 + threadIdx.x + qn * BLOCK;
            okn              = channel_rows<PART>(plan, pb, cn, rn, BLOCK, in_tile(qn, per, rn, BLOCK, n), vn);
          }
        }
        unsigned char* dst = smem + tl.val_off[c];
#define GBX_STAGE(T)                                                                           \
  _Pragma("unroll") for (int q = 0; q < kBatch; ++q) if ((rows >> q) & 1u)                     \
    reinterpret_cast<T*>(dst)[pos[q]] = static_cast<T>(v[q]);                                  \
  break;
        switch (pt_width(plan.chan[c].ptype)) {
          case 1: GBX_STAGE(uint8_t)
          case 2: GBX_STAGE(uint16_t)
          case 4: GBX_STAGE(uint32_t)
          default: GBX_STAGE(uint64_t)
        }
#undef GBX_STAGE
        if (tl.ok_off[c] != 0) {
          uint8_t* d = smem + tl.ok_off[c];
#pragma unroll
          for (int q = 0; q < kBatch; ++q)
            if ((rows >> q) & 1u) d[pos[q]] = (ok >> q) & 1u;
        }
#pragma unroll
        for (int q = 0; q < kBatch; ++q) v[q] = vn[q];
        ok = okn;
      }
    }
    if (nspill != 0) spill_rows<NW, PART>(plan, t, pb, spill, nspill, t0, max_probes);
    __syncthreads();
    // 4. one chunk per thread
    const uint32_t nchunks = total >> 16;
    for (uint32_t c0 = static_cast<uint32_t>(warp) * 32; c0 < nchunks; c0 += BLOCK) {
      const uint32_t ci  = c0 + lane;
      const bool active  = ci < nchunks;
      const uint32_t s   = cslot[active ? ci : c0];
      const uint32_t o0  = oc[s];
      const uint32_t j0  = (ci - (o0 >> 16)) * kChunk;
      const uint32_t p0  = (o0 & 0xffffu) + j0;
      const uint32_t len = min(static_cast<uint32_t>(kChunk), (oc[s + 1] & 0xffffu) - p0);
      const uint32_t s0  = __shfl_sync(kFull, s, 0);
      const uint32_t lanes = __ballot_sync(kFull, active);
      const bool uniform   = __all_sync(kFull, active && s == s0);
      if (!active) continue;
      for (int c = 0; c < plan.nchan; ++c) {
        const Channel& ch = plan.chan[c];
#define GBX_FOLD(P) fold_chunk<P>(ch, smem, sl, tl.val_off[c], tl.ok_off[c], p0, len, s, uniform, lanes, t.status); break;
        switch (ch.ptype) {
          case P_I8: GBX_FOLD(P_I8)
          case P_I16: GBX_FOLD(P_I16)
          case P_I32: GBX_FOLD(P_I32)
          case P_I64: GBX_FOLD(P_I64)
          case P_U8: GBX_FOLD(P_U8)
          case P_U16: GBX_FOLD(P_U16)
          case P_U32: GBX_FOLD(P_U32)
          case P_U64: GBX_FOLD(P_U64)
          case P_F32: GBX_FOLD(P_F32)
          case P_F64: GBX_FOLD(P_F64)
          default: GBX_FOLD(P_BOOL)
        }
#undef GBX_FOLD
      }
    }
    // no barrier here: the next tile's ranking touches only the keys and
    // `cnt`, and its scan waits for every thread to have left this fold
  }
  __syncthreads();
  // merge the CTA's table into the global one
  const Level<Shared> L{static_cast<uint32_t>(__cvta_generic_to_shared(smem)), &sl};
  const Level<Global> G = global_level(t);
  for (uint32_t s = threadIdx.x; s <= S; s += BLOCK) {
    if (srows[s] == 0) continue;
    uint64_t k[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) k[w] = skeys[s * NW + w];
    const int64_t g = global_slot<NW>(t, k, max_probes);
    if (g >= 0) merge_slot<Shared>(plan, L, s, G, g, t.status);
  }
}

template <int NW, bool PART, int BLOCK>
cudaError_t launch_tiled_as(const Plan& p, const TableRef& t, const SmemLayout& sl, const TiledLayout& tl, int64_t n,
                            const PartBufs& pb, const uint32_t* n_part, int num_sms, uint32_t smem_probes,
                            uint32_t max_probes, cudaStream_t st)
{
  const void* fn = reinterpret_cast<const void*>(k_agg_tiled<NW, PART, BLOCK>);
  cudaError_t e  = ensure_dynamic_smem(fn, tl.total);
  if (e != cudaSuccess) return e;
  const int64_t ntiles = (n + tl.tile_rows - 1) / tl.tile_rows;
  const int64_t cap    = static_cast<int64_t>(num_sms) * (1024 / BLOCK);
  const int grid       = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(ntiles, cap)));
  k_agg_tiled<NW, PART, BLOCK><<<grid, BLOCK, tl.total, st>>>(p, t, sl, tl, n, pb, n_part, smem_probes, max_probes);
  return cudaGetLastError();
}

template <bool PART>
cudaError_t launch_tiled(const Plan& p, const TableRef& t, const SmemLayout& sl, int64_t n, const PartBufs& pb,
                         const uint32_t* n_part, int num_sms, uint32_t smem_probes, uint32_t max_probes,
                         cudaStream_t st)
{
  TiledLayout tl = pick_tiled_layout(sl, p);
  if (tl.tile_rows == 0) return cudaErrorInvalidValue;
  if (n <= 0) return cudaSuccess;
  // few rows: tiles small enough that every SM gets one
  const int64_t ctas = static_cast<int64_t>(num_sms) * (1024 / tl.block);
  const int64_t want = (n + ctas * tl.block - 1) / (ctas * tl.block) * tl.block;
  if (want < tl.tile_rows) tl = tiled_layout(sl, p, tl.block, static_cast<int>(want));
  const bool one = p.key.nwords == 1;
  if (tl.block == 512)
    return one ? launch_tiled_as<1, PART, 512>(p, t, sl, tl, n, pb, n_part, num_sms, smem_probes, max_probes, st)
               : launch_tiled_as<2, PART, 512>(p, t, sl, tl, n, pb, n_part, num_sms, smem_probes, max_probes, st);
  return one ? launch_tiled_as<1, PART, 1024>(p, t, sl, tl, n, pb, n_part, num_sms, smem_probes, max_probes, st)
             : launch_tiled_as<2, PART, 1024>(p, t, sl, tl, n, pb, n_part, num_sms, smem_probes, max_probes, st);
}

}  // namespace

bool tiled_fits(const SmemLayout& sl, const Plan& p, bool two_per_sm)
{
  if (sl.slots > static_cast<uint32_t>(kMaxSlots)) return false;
  const TiledLayout tl = pick_tiled_layout(sl, p);
  return tl.tile_rows > 0 && (!two_per_sm || tl.block == 512);
}

int tiled_rows(const SmemLayout& sl, const Plan& p)
{
  return sl.slots > static_cast<uint32_t>(kMaxSlots) ? 0 : pick_tiled_layout(sl, p).tile_rows;
}

cudaError_t launch_agg_tiled(const Plan& p, const TableRef& t, const SmemLayout& sl, int64_t n, int num_sms,
                             uint32_t smem_probes, uint32_t max_probes, cudaStream_t st)
{
  return launch_tiled<false>(p, t, sl, n, PartBufs{}, nullptr, num_sms, smem_probes, max_probes, st);
}

cudaError_t launch_agg_tiled_part(const Plan& p, const TableRef& t, const SmemLayout& sl, const PartBufs& in,
                                  const uint32_t* n_rows, int64_t n, int num_sms, uint32_t smem_probes,
                                  uint32_t max_probes, cudaStream_t st)
{
  return launch_tiled<true>(p, t, sl, n, in, n_rows, num_sms, smem_probes, max_probes, st);
}

}  // namespace gbx
