// gbx_join.hpp -- the join over packed one-word keys (gbx_join_packed.cu),
// which gbx_hash_join (gbx_join.cu) tries first.
#pragma once

#include "gbx_host.hpp"

namespace gbx {

// Joins `probe` against `build` (sizes, types and kind checked by the caller)
// when both are non-empty and the key packs into one 64-bit word; false
// (nothing done) otherwise.  The gather maps go to out_probe / out_build
// (which the caller releases after a failure); the stream is synchronised
// before it returns true.
bool packed_join(const gbx_table_view* build, const gbx_table_view* probe, int32_t compare_nulls, int32_t kind,
                 Alloc& a, gbx_column& out_probe, gbx_column& out_build);

}  // namespace gbx
