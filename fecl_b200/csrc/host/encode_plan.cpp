#include "encode_plan.hpp"

#include <algorithm>

namespace fecl {

LdpcEncodePlan build_ldpc_encode_plan(const LdpcCode& code, uint32_t max_bytes) {
  LdpcEncodePlan p;
  const uint32_t K = code.msg_size();
  const Csr &A = code.gen_a(), &B = code.gen_b(), &T = code.gen_t();
  const uint32_t gap = code.gen_dc().rows, rows = A.rows;
  auto up16 = [](uint64_t x) { return (x + 15) & ~uint64_t(15); };
  const uint64_t off_gap = up16(uint64_t(K) + 1), off_t = up16(off_gap + gap), bytes = up16(off_t + rows) + 16;
  if (bytes > max_bytes || T.rows != rows || B.rows != rows || uint64_t(K) + gap + rows != code.parity_size()) return p;
  p.zero_at = K;
  p.off_gap = uint32_t(off_gap);
  p.off_t = uint32_t(off_t);
  p.bytes = uint32_t(bytes);

  // T is stored by column: entry list r begins with r itself, the rest are the rows that
  // parity bit r adds into
  std::vector<uint32_t> level(rows, 0), sources(rows, 0);
  p.chain = true;
  for (uint32_t r = 0; r < rows; ++r) {
    const uint32_t b = T.row_ptr[r], e = T.row_ptr[r + 1];
    if (b == e || T.col_idx[b] != r) return p;
    const bool next_alone = r + 1 < rows ? (e - b == 2 && T.col_idx[b + 1] == r + 1) : e - b == 1;
    if (!next_alone) p.chain = false;
    for (uint32_t k = b + 1; k < e; ++k) {
      const uint32_t i = T.col_idx[k];
      if (i <= r || i >= rows) return p;
      level[i] = std::max(level[i], level[r] + 1);
      ++sources[i];
    }
  }
  for (uint32_t c : B.col_idx)
    if (c >= gap) return p;

  p.row_ptr.push_back(0);
  for (uint32_t r0 = 0; r0 < rows; r0 += 32) {
    uint32_t d = 0;
    for (uint32_t r = r0; r < std::min(rows, r0 + 32); ++r)
      d = std::max(d, A.row_ptr[r + 1] - A.row_ptr[r] + B.row_ptr[r + 1] - B.row_ptr[r]);
    const size_t at = p.row_idx.size();
    p.row_idx.resize(at + size_t(d) * 32, p.zero_at);
    for (uint32_t r = r0; r < std::min(rows, r0 + 32); ++r) {
      size_t k = at + (r - r0);
      for (uint32_t e = A.row_ptr[r]; e < A.row_ptr[r + 1]; ++e, k += 32) p.row_idx[k] = A.col_idx[e];
      for (uint32_t e = B.row_ptr[r]; e < B.row_ptr[r + 1]; ++e, k += 32) p.row_idx[k] = p.off_gap + B.col_idx[e];
    }
    p.row_ptr.push_back(uint32_t(p.row_idx.size()));
  }
  p.ok = true;
  if (p.chain) return p;

  const uint32_t depth = rows ? *std::max_element(level.begin(), level.end()) : 0;
  std::vector<uint32_t> count(depth + 2, 0), place(rows, 0);
  for (uint32_t r = 0; r < rows; ++r)
    if (level[r]) ++count[level[r]];
  p.level_ptr.assign(depth + 1, 0);  // levels 1 .. depth
  for (uint32_t l = 1; l <= depth; ++l) p.level_ptr[l] = p.level_ptr[l - 1] + count[l];
  p.level_rows.resize(p.level_ptr[depth]);
  std::vector<uint32_t> fill(p.level_ptr.begin(), p.level_ptr.end());
  for (uint32_t r = 0; r < rows; ++r)
    if (level[r]) p.level_rows[place[r] = fill[level[r] - 1]++] = r;
  p.src_ptr.assign(p.level_rows.size() + 1, 0);
  for (size_t q = 0; q < p.level_rows.size(); ++q) p.src_ptr[q + 1] = p.src_ptr[q] + sources[p.level_rows[q]];
  p.src_idx.resize(p.src_ptr.back());
  std::vector<uint32_t> at(p.src_ptr.begin(), p.src_ptr.end() - 1);
  for (uint32_t r = 0; r < rows; ++r)
    for (uint32_t k = T.row_ptr[r] + 1; k < T.row_ptr[r + 1]; ++k) p.src_idx[at[place[T.col_idx[k]]]++] = r;
  return p;
}

}  // namespace fecl
