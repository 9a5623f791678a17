// gbx_rows.cuh -- a thread's rows taken several at a time: keys packed and
// values loaded column by column, so that one uniform branch on a column's
// width (and one look at its descriptor) serves PER rows and their loads are
// in flight together.
#pragma once

#include "gbx_device.cuh"

namespace gbx {
namespace dev {

// Packed keys of rows r0 + q * step for the bits q set in `kept` (the layout
// of pack_key_from, gbx_device.cuh); returns the rows not excluded by
// null_policy::EXCLUDE.
template <int PER, int NW, class Bufs>
__device__ __forceinline__ uint32_t pack_rows(const KeyPlan& kp, const Bufs& bufs, int64_t r0, int step, uint32_t kept,
                                              uint64_t (&k)[PER][NW])
{
#pragma unroll
  for (int q = 0; q < PER; ++q)
#pragma unroll
    for (int w = 0; w < NW; ++w) k[q][w] = 0;
  for (int c = 0; c < kp.ncols; ++c) {
    const KeyCol& kc     = kp.cols[c];
    const int64_t i0     = r0 + bufs.offset(c);
    const uint32_t* mask = bufs.mask(c);
    uint32_t nulls       = 0;
    if (mask != nullptr) {
#pragma unroll
      for (int q = 0; q < PER; ++q)
        if (((kept >> q) & 1u) && !bit_valid(mask, i0 + static_cast<int64_t>(q) * step)) nulls |= 1u << q;
      if (kp.skip_null_rows) {
        kept &= ~nulls;
        nulls = 0;
      }
    }
    const uint32_t load = kept & ~(kc.null_bit ? nulls : 0u);
    uint64_t v[PER];
    switch (kc.width) {
#define GBX_LOAD_KEYS(T)                                                                                  \
  {                                                                                                       \
    const T* p = reinterpret_cast<const T*>(bufs.data(c)) + i0;                                           \
    _Pragma("unroll") for (int q = 0; q < PER; ++q)                                                       \
      v[q] = ((load >> q) & 1u) ? static_cast<uint64_t>(__ldg(p + static_cast<int64_t>(q) * step)) : 0;   \
  }                                                                                                       \
  break;
      case 1: GBX_LOAD_KEYS(uint8_t)
      case 2: GBX_LOAD_KEYS(uint16_t)
      case 4: GBX_LOAD_KEYS(uint32_t)
      default: GBX_LOAD_KEYS(unsigned long long)
#undef GBX_LOAD_KEYS
    }
    if (kc.is_float) {
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        if (kc.width == 4) {
          const float f = __uint_as_float(static_cast<uint32_t>(v[q]));
          if (f != f) v[q] = 0x7fc00000u;
          else if (f == 0.0f) v[q] = 0;
        } else {
          const double d = __longlong_as_double(static_cast<long long>(v[q]));
          if (d != d) v[q] = 0x7ff8000000000000ULL;
          else if (d == 0.0) v[q] = 0;
        }
      }
    } else if (kc.is_bool) {
#pragma unroll
      for (int q = 0; q < PER; ++q) v[q] = v[q] != 0;
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const uint64_t x = v[q] << kc.shift;
      if constexpr (NW == 1) {
        k[q][0] |= x;
      } else {
        k[q][0] |= kc.word == 0 ? x : 0;
        k[q][1] |= kc.word == 0 ? 0 : x;
      }
    }
    if (kc.null_bit) {
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const uint64_t x = ((nulls >> q) & 1u) ? 1ULL << kc.null_shift : 0;
        if constexpr (NW == 1) {
          k[q][0] |= x;
        } else {
          k[q][0] |= kc.null_word == 0 ? x : 0;
          k[q][1] |= kc.null_word == 0 ? 0 : x;
        }
      }
    }
  }
  return kept;
}

// Elements i0 + q * step of a column of `width`-byte elements for the bits q
// set in `rows` (0 for the others).
template <int PER>
__device__ __forceinline__ void load_rows(int width, const void* data, int64_t i0, int step, uint32_t rows,
                                          uint64_t (&v)[PER])
{
  switch (width) {
#define GBX_LOAD_ROWS(T)                                                                                  \
  {                                                                                                       \
    const T* p = reinterpret_cast<const T*>(data) + i0;                                                   \
    _Pragma("unroll") for (int q = 0; q < PER; ++q)                                                       \
      v[q] = ((rows >> q) & 1u) ? static_cast<uint64_t>(__ldg(p + static_cast<int64_t>(q) * step)) : 0;   \
  }                                                                                                       \
  break;
    case 1: GBX_LOAD_ROWS(uint8_t)
    case 2: GBX_LOAD_ROWS(uint16_t)
    case 4: GBX_LOAD_ROWS(uint32_t)
    default: GBX_LOAD_ROWS(unsigned long long)
#undef GBX_LOAD_ROWS
  }
}

// The bits q of `rows` whose element i0 + q * step is valid.
template <int PER>
__device__ __forceinline__ uint32_t valid_rows(const uint32_t* mask, int64_t i0, int step, uint32_t rows)
{
  if (mask == nullptr) return rows;
  uint32_t ok = 0;
#pragma unroll
  for (int q = 0; q < PER; ++q)
    if (((rows >> q) & 1u) && bit_valid(mask, i0 + static_cast<int64_t>(q) * step)) ok |= 1u << q;
  return ok;
}

// A 32-bit mix of a packed key for a table of the CTA's own (any mix will do
// there; the global table's 64-bit hash costs about twice as much): the words
// combined with odd constants, then the 32-bit finaliser of MurmurHash3
// (Appleby, public domain).
template <int NW>
__device__ __forceinline__ uint32_t tile_hash(const uint64_t (&k)[NW])
{
  uint32_t h = static_cast<uint32_t>(k[0]) ^ (static_cast<uint32_t>(k[0] >> 32) * 0x9e3779b1u);
  if constexpr (NW == 2)
    h = (h * 0x85ebca6bu) ^ static_cast<uint32_t>(k[1]) ^ (static_cast<uint32_t>(k[1] >> 32) * 0xc2b2ae35u);
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return h;
}

// Slots of a batch of keys in a CTA table of `mask + 1` slots at `skeys`
// (shared address keys_sa), inserting absent keys.  The home slots are read
// together; rows whose home slot does not hold their key probe on one after
// another, and the warp meets again after each: without that, the lanes that
// leave a probe loop at different times run everything after it apart.  All
// 32 lanes call it.  Returns the rows that found a slot (slot[q] = `mask + 1`
// for the all-ones key, which has the reserved slot).
template <int PER, int NW>
__device__ __forceinline__ uint32_t find_slots(uint64_t* skeys, uint32_t keys_sa, uint32_t mask, uint32_t kept,
                                               const uint64_t (&k)[PER][NW], uint32_t max_probes,
                                               uint32_t (&slot)[PER])
{
  uint32_t found = 0;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    slot[q]  = tile_hash<NW>(k[q]) & mask;
    bool hit = true;
#pragma unroll
    for (int w = 0; w < NW; ++w) hit = hit && skeys[slot[q] * NW + w] == k[q][w];
    // a key with an all-ones word may match a slot being written: find_or_insert settles it
    if constexpr (NW == 2) hit = hit && k[q][0] != kEmptyWord && k[q][1] != kEmptyWord;
    // an all-ones key also matches an empty slot: it takes the reserved one
    if (key_is_empty<NW>(k[q])) {
      slot[q] = mask + 1;
      hit     = true;
    }
    found |= hit ? 1u << q : 0u;
  }
  found &= kept;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    if (((kept & ~found) >> q) & 1u) {
      uint32_t s = slot[q];
      int at     = -1;
      if constexpr (NW == 1) {
        for (uint32_t p = 0; p < max_probes; ++p) {
          // plain loads: a stale read of an empty slot is settled by the
          // compare-and-swap
          const uint64_t cur = skeys[s];
          if (cur == k[q][0]) {
            at = static_cast<int>(s);
            break;
          }
          if (cur == kEmptyWord) {
            const unsigned long long old =
              atomicCAS(reinterpret_cast<unsigned long long*>(skeys + s), static_cast<unsigned long long>(kEmptyWord),
                        static_cast<unsigned long long>(k[q][0]));
            if (old == kEmptyWord || old == k[q][0]) {
              at = static_cast<int>(s);
              break;
            }
          }
          s = (s + 1) & mask;
        }
      } else {
        at = static_cast<int>(find_or_insert<Shared, NW>(keys_sa, mask, k[q], s, max_probes));
      }
      if (at >= 0) {
        slot[q] = static_cast<uint32_t>(at);
        found |= 1u << q;
      }
    }
    __syncwarp();
  }
  return found;
}

}  // namespace dev
}  // namespace gbx
