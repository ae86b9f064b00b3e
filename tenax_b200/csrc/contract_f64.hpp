// One-launch FP64 contraction (contract_f64.cu): its tables and launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <map>
#include <utility>
#include <vector>

namespace tnx {

// One (A block, B block) pair of an output block.  An axis maps an index to an
// element offset inside its block: index * str, or tab[index] where `*_tab` is
// the first entry of a table (>= 0).
struct ContractSpan {
  int64_t a_off, b_off;  // element offsets of the two blocks
  int32_t ar_tab, ar_str, ak_tab, ak_str;
  int32_t br_tab, br_str, bk_tab, bk_str;
  int32_t K, a_slot, b_slot, pad;  // slots of the operand pointer tables, where the launch has them
};
static_assert(sizeof(ContractSpan) == 64, "read as four 16-byte units");

struct ContractTile {
  int64_t out_off;        // element offset of the output block
  int32_t M, N, m0, n0;   // the block's extents, the tile's origin
  int32_t span0, nspan, ktiles;  // pairs summed; 16-deep K tiles of all of them
  int32_t r_tab, r_str, c_tab, c_str;
  int32_t out_slot;  // slot of the output pointer table, where the launch has one
  double scale;      // the result's factor
};
static_assert(sizeof(ContractTile) == 64, "one record a tile");

// Offset tables of one step's axes: an axis of legs (extent, stride), outermost
// first, is affine where the legs merge into one stride, and otherwise a table
// shared by every axis of the same legs.
struct AxisTabs {
  // entries of all tables (they are indexed by int32_t); a step that needs more
  // takes the packed path, whose tables do not grow with the extents
  int64_t limit = INT32_MAX;
  std::vector<int32_t> tab;
  std::map<std::vector<std::pair<int64_t, int64_t>>, int32_t> seen;
  // false, with nothing filled: beyond the limit
  bool add(const std::vector<std::pair<int64_t, int64_t>>& legs, int32_t* t, int32_t* str) {
    std::vector<std::pair<int64_t, int64_t>> m;
    for (const auto& l : legs) {
      if (l.first == 1) continue;
      if (!m.empty() && m.back().second == l.first * l.second)
        m.back() = {m.back().first * l.first, l.second};
      else
        m.push_back(l);
    }
    *t = -1;
    *str = m.empty() ? 0 : static_cast<int32_t>(m[0].second);
    if (m.size() < 2) return true;
    *str = static_cast<int32_t>(m.back().second);
    auto it = seen.find(m);
    if (it == seen.end()) {
      int64_t n = 1;
      for (const auto& l : m) n *= l.first;
      if (static_cast<int64_t>(tab.size()) + n > limit) return false;
      it = seen.emplace(m, static_cast<int32_t>(tab.size())).first;
      const size_t first = tab.size();
      tab.resize(first + static_cast<size_t>(n));
      // the innermost leg, then that pattern shifted by each outer leg in turn
      int64_t len = 1;
      for (size_t l = m.size(); n > 0 && l-- > 0; len *= m[l].first)
        for (int64_t k = 1; k < m[l].first; ++k)
          for (int64_t i = 0; i < len; ++i)
            tab[first + k * len + i] = tab[first + i] + static_cast<int32_t>(k * m[l].second);
    }
    *t = it->second;
    return true;
  }
};

// The kernel forms the offsets inside a tile, up to 16 K steps and 128 rows, in
// 32 bits.  Blocks of fewer than 2^31 elements cannot leave that range; for
// larger ones these are the K steps a span and the rows an output matrix may
// have, given the longest stride of either.
constexpr int64_t kTileK = 16, kTileRows = 128;
inline int64_t span_k(int64_t K, int64_t stride) {
  return (kTileK - 1) * stride <= INT32_MAX ? K : INT32_MAX / stride + 1;
}
inline int64_t matrix_rows(int64_t M, int64_t stride) {
  return (kTileRows - 1) * stride <= INT32_MAX ? M : INT32_MAX / stride + 1;
}

// an output block as the choice of tile shape sees it
struct ContractBlk {
  int64_t M, N, ktiles, k4;  // k4: 4-deep K steps of all pairs
};

struct ContractLaunch {
  const double *a, *b;
  double* c;
  // batched launches: base addresses by slot instead of a, b and c (nullptr: the single base)
  const uint64_t *a_ptrs, *b_ptrs, *c_ptrs;
  const int32_t* skip;  // nonzero on the device: do nothing
  const ContractTile* tiles;
  const ContractSpan* spans;
  const int32_t* tab;
  int n_tiles, shape;
  int split, parts;  // K shares of one cluster, and clusters per output tile
  bool a_kfast, b_kfast;  // whether K is the fast axis of the operand's blocks
  // whether pairs of the fast axis may be read by 16 bytes, given a base on 16
  // bytes (a batched launch's bases and block offsets are on 16 bytes)
  bool a_vec, b_vec;
};

constexpr int kContractShapes = 4;
// between min_split and max_split K shares; 8 keeps them in one cluster (no
// workspace, no second launch).  A block's sums depend on the shares alone, not
// on the tile shape.
void contract_choose(const std::vector<ContractBlk>& blks, int n_sm, int min_split, int max_split, int* shape,
                     int* split, int* parts);
// appends to `dst` the tiles of the blocks `proto` (M, N and the block's axes
// set) in the launch's shape, longest first to within 1/32; returns their number
int64_t contract_tiles(const std::vector<ContractTile>& proto, const std::vector<ContractBlk>& blks, int shape,
                       std::vector<uint8_t>& dst);
cudaError_t launch_contract_f64(const ContractLaunch& L, cudaStream_t st);

}  // namespace tnx
