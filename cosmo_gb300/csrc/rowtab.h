// Rows of a stored H from sorted move tables (bitstring, untruncated bases
// whose species each have one parity).
//
// hbuild.cu's general builder lets one thread enumerate the moves of one row
// twice (count, fill) and sorts every row afterwards.  Here the moves are
// tabulated once per species configuration, sorted by target: per neutron block
// its target blocks (one or two neutrons moved), per proton configuration its
// one-proton moves by change of 2m and its moves within the block.  A row is
// then the merge of short lists that are already in column order.
#pragma once
#include "device.h"

namespace cg {

// Column-ordered rows; count() then fill(), on stream s.  Null from
// row_tables() where the general builder has to serve.
struct RowTables {
  virtual ~RowTables() = default;
  // elements of every row (|value| >= 1e-14); false when a row is too long for fill()
  virtual bool count(uint32_t* counts) = 0;
  // columns and values (out64, or hi + lo) at rowptr, the diagonal, and the
  // number of entries on or above it
  virtual void fill(const uint64_t* rowptr, uint32_t* col, double* out64, float* hi, float* lo, double* diag,
                    unsigned long long* upper) = 0;
};
std::unique_ptr<RowTables> row_tables(const Basis& b, const DevOperator& op, cudaStream_t s);

}  // namespace cg
