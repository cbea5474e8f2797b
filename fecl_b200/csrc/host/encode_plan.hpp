// Tables of the device LDPC encoder (device/encode.cu), built from the generator
// pieces of LdpcCode::encode.
#pragma once

#include <cstdint>
#include <vector>

#include "codes.hpp"

namespace fecl {

// One frame's bytes in the encoder's shared memory: the message at [0, K), a zero at
// zero_at (what padding entries read), the gap parity from off_gap and the T-part
// parity from off_t; both offsets are multiples of 16.
struct LdpcEncodePlan {
  bool ok = false;  // false: a T part that is not lower triangular, or a frame beyond shared memory
  uint32_t zero_at = 0, off_gap = 0, off_t = 0, bytes = 0;
  // T-part rows (A and B columns together), 32 rows to a block: block b's entry j of row
  // 32 b + l is row_idx[row_ptr[b] + 32 j + l], short rows filled up with zero_at, so that a warp
  // reads a block's entries as contiguous lines.
  std::vector<uint32_t> row_ptr, row_idx;
  // Back substitution through T.  chain: every parity bit adds into the next one alone
  // (the accumulator of the DVB-S2 codes).  Otherwise rows by level -- a row's sources
  // all lie in lower levels -- position q holding row level_rows[q], whose sources are
  // src_idx[src_ptr[q] .. src_ptr[q + 1]).  Level 0, which has none, is left out.
  bool chain = false;
  std::vector<uint32_t> level_ptr, level_rows, src_ptr, src_idx;
};

LdpcEncodePlan build_ldpc_encode_plan(const LdpcCode& code, uint32_t max_bytes);

}  // namespace fecl
