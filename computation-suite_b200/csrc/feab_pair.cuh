// Pair records of a tile operator: the operand layout of the block SpMM on the FP64 tensor path.
//
// A tile's groups are taken two at a time (pair q: groups 2 (q % 2) and the next of tile q / 2); the up
// to six rows of a pair are the rows of an 8 x 4 operand of mma.sync.m8n8k4, and the sorted union of
// the two column lists is walked four columns at a time.  A record holds one such step: the
// operand's six rows (row k, column t at 4 k + t, so that lane l = 4 k + t of a warp reads its own
// element) and the four columns.  Consecutive nodes of a structured hex8 mesh share 18 of their 27
// neighbours, so a pair has 108 columns and 56 % of the tensor work is on nonzeros.
#pragma once
#include "feab_common.cuh"

namespace feab {

// The least panel width that is multiplied through pair records: a tile of mma.sync.m8n8k4 is 8 columns.  The
// records take 27 steps of 208 bytes per pair of nodes of a structured mesh, 2.8 KB per node beside the 1.9 KB
// of its CSR values, and are not made for narrower panels.
constexpr int kPairPanel = 8;

struct __align__(16) PairRecord {
  double val[24];
  int32_t col[4];
};
static_assert(sizeof(PairRecord) == 208, "13 words of 16 bytes");

struct PairView {
  const int32_t* off;      // 2 n_tiles + 1: first record of each pair (NULL: the operator has none)
  const PairRecord* rec;
};

// The section behind the operator's other arrays: the offsets, then the records.
inline size_t pair_offset_bytes(int32_t n_tiles) {
  return (sizeof(int32_t) * (2 * (size_t)n_tiles + 1) + 255) & ~size_t(255);
}
inline size_t pair_section_bytes(int32_t n_tiles, int64_t steps) {
  return pair_offset_bytes(n_tiles) + sizeof(PairRecord) * (size_t)steps;
}
// `reserved` of the operator is the section's place, in units of 256 bytes from tile_g0, the storage's
// first array (0: an operator without pair records).
inline PairView pair_view(const feab_tile_operator* T) {
  if (!T || T->reserved <= 0) return PairView{nullptr, nullptr};
  const char* p = reinterpret_cast<const char*>(T->tile_g0) + 256 * (size_t)T->reserved;
  return PairView{reinterpret_cast<const int32_t*>(p),
                  reinterpret_cast<const PairRecord*>(p + pair_offset_bytes(T->n_tiles))};
}

}  // namespace feab
