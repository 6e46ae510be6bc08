// Stored rows in tiles of 32: the assembled form of operators whose adjoint
// products are site pairs (Heisenberg, XXZ, J1-J2, XY, DM, Ising chains) on
// u64 states, in any sector.
//
// Tile t holds rows 32 t .. 32 t + 31, one lane per row: entry slot j of row
// 32 t + l is entries[(tile_ptr[t] + j) * 32 + l], so a warp reads a slot as
// one 128-byte line and needs no row pointers and no sums across lanes. Rows
// list their transitions from the highest flipped bond down. Consecutive rows
// share their high bits, so the lanes of a slot mostly hop the same bond and
// their columns lie close together. An entry is
//   column | code << col_bits,  code = (amplitude * phases + phase) * classes + orbit class,
// with 0xffffffff in unused slots. The code tables hold the entry's value
// without the orbit factor (block action, coordinates x / sqrt(R)) and divided
// by sqrt(R_column) (y = H x), so neither action needs a scaled copy of x.
// Transitions of a row that meet in one column stay separate entries, or none
// when they cancel.
#pragma once

#include <cstdint>

#include "basis.cuh"
#include "hv_tile.cuh"

namespace qmbed {

struct TileRows {
  uint64_t n = 0;
  int sms = 0;              // of the device
  bool complex_values = false;
  int col_bits = 0, codes = 0;
  uint64_t nnz = 0;         // off-diagonal nonzeros after coalescing
  int distinct_values = 0;  // distinct coalesced values (real operators)
  DeviceBuffer tile_ptr;    // u32, tiles + 1, in slots of 32 entries
  DeviceBuffer entries;
  DeviceBuffer values;      // per code: (re, im) FP64, then (re, im) / sqrt(R)
  DeviceBuffer diag64, diag32;
};

// Assembles `prog` (adjoint products, not uploaded) on `basis`. Returns false,
// with `out` unspecified, when the operator is outside this form: u128
// states, products that flip or read more than two sites with a flip, more
// than 64 transitions in one row, or codes that do not fit beside the column.
bool assemble_tile_rows(const SpinBasis& basis, const FlipProgram& prog, bool real, TileRows& out);

// y = H x. Real rows take real or interleaved complex vectors, complex rows
// complex ones. sqrt_table: [257 + R] sqrt(R).
void tile_spmv(const TileRows& rows, const SpinBasis& basis, const double* sqrt_table, int precision,
               bool complex_vectors, const void* x, void* y, cudaStream_t stream);

// out = alpha (S^-1 H S) z + beta z + gamma p on row-major n x nb blocks (real
// rows; nb = 8 or 16; p may be null; out may alias p, not z).
constexpr int kTileBlockShapes = 4;
void tile_spmm(const TileRows& rows, int shape, int precision, int nb, const void* z, const void* p, void* out,
               double alpha, double beta, double gamma, cudaStream_t stream);

}  // namespace qmbed
