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
// Whether tables of `bytes` (while they are made; about half afterwards) pay
// whose entries are read `uses` times by all rows together.  With one species
// moving the lists are as long as the rows themselves and no two rows share one
// (30 states, 10 protons: 32 bytes for each of 7e8 elements), and the general
// builder, whose unsorted values take 8 bytes an element, needs less memory.
constexpr uint64_t kRowTableBytes = 1ull << 30;
inline bool row_tables_worth(uint64_t bytes, uint64_t uses) { return bytes <= kRowTableBytes + 8 * uses; }
std::unique_ptr<RowTables> row_tables(const Basis& b, const DevOperator& op, cudaStream_t s);

}  // namespace cg
