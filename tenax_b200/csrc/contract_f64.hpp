// One-launch FP64 contraction (contract_f64.cu): its tables and launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

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
// set) in the launch's shape, longest first; returns their number
int64_t contract_tiles(const std::vector<ContractTile>& proto, const std::vector<ContractBlk>& blks, int shape,
                       std::vector<uint8_t>& dst);
cudaError_t launch_contract_f64(const ContractLaunch& L, cudaStream_t st);

}  // namespace tnx
