// Factored H + lambda * J-J+ product: the two-body operator applied through
// cores, the determinants with two particles taken out.
//
// Every matrix element between determinants that differ by at most two moves
// is a sum over the pairs of particles the operator acts on.  With the
// one-body terms spread over those pairs, H = sum over species pairs of
//   y[K + cd] += s_cd sum_ab V[cd][ab] s_ab x[K + ab],
// where K runs over the cores (a determinant without one neutron and one
// proton, without two neutrons, or without two protons), ab and cd over the
// pairs of one channel (2m and parity that K lacks), V is one small symmetric
// matrix per channel and s_ab the fermion phase of adding the pair to K.  A
// core reads each of its rows of x once for all its outputs, so a product
// takes k_n k_p + k_n (k_n - 1) / 2 + k_p (k_p - 1) / 2 row reads per
// determinant instead of one per matrix element (28 instead of 637 on the
// fp shell with 4 + 4 particles), and the element sums become small dense
// matrix products.  The reference applies the same terms one element at a
// time (SM::PPMatrix::TimesVectorSymmetric, include/sm/PPMatrix.cxx:117-152).
#pragma once
#include <cstdint>
#include <memory>
#include <vector>

#include "device.h"

namespace cg {

// one CTA's work: all spectators of one core (or neutron core) and channel
struct FJob {
  uint32_t list;   // first entry of its pairs in FactoredOp::list
  uint32_t npair;  // pairs the core has room for
  uint32_t spect;  // kind 0: first spectator core; kind 1: first entry of FactoredOp::spect, or ~0u: rows first, first + 1, ..
  uint32_t count;  // spectators
  uint32_t w0;     // first value of the channel's matrix
  uint32_t ldw;    // its order
  uint32_t kind;   // 0: neutron + proton pairs; 1: pairs of one species
  uint32_t first;
};
static_assert(sizeof(FJob) == 32, "FJob layout");

// One pair of a job: the first row (neutrons) or rank (protons) of core +
// pair, and packed: position in the channel | spectator state << 8 | slot << 16 |
// phase << 31 (slot and phase without the part the spectator adds).
struct FPair {
  uint32_t row, meta;
};

struct FactoredOp {
  uint64_t n = 0;
  int cols = 0;                 // s.p. states of the spectators' species
  int slots = 0;                // partial sums per row: kn kp + kn (kn - 1) / 2 + kp (kp - 1) / 2
  int smem32 = 0;               // shared memory of k_fact32
  int dmax = 0;                 // most pairs of one job
  int dmax_same = 0;            // of a job of one species
  uint64_t njobs = 0, njobs_pn = 0;  // jobs, of which (the first) neutron + proton pairs
  double macs = 0, macs_same = 0;  // multiply-adds per vector of one product, tiles filled up
  DBuf<FJob> jobs;              // largest first
  DBuf<FPair> list;
  DBuf<uint32_t> stab;          // spectator core x cols: row offset of core + state | position << 27, ~0u if none
  DBuf<uint32_t> spect;         // block starts of each proton class
  double est_us = 0;            // estimated time of one product
  DBuf<float> wf;               // channel matrices
  mutable DBuf<unsigned char> z;  // partial sums: slots x n rows of 32 bytes (factored_ready)
  uint64_t bytes() const {
    return jobs.bytes() + list.bytes() + stab.bytes() + spect.bytes() + wf.bytes() + z.bytes();
  }
};

// Tables of the factored product, or null where it does not apply (a truncated
// or wide basis, a species without particles, channels, rows or a work area
// beyond its limits), where its tables cannot be allocated, or where it is
// estimated slower than other_us, the time of the product it would replace.
std::shared_ptr<FactoredOp> factored_build(const System& sys, const Operator& op, const Basis& b, double other_us,
                                           cudaStream_t s);
constexpr uint64_t kFactoredMaxWork = 32ull << 30;
// stored matrices of fewer entries keep the row-wise product without an estimate
// (fp 2+4, 3.3e7 entries: 120 us row-wise, 60 factored; sd 4+4, 6e6: 24 and 33)
constexpr uint64_t kFactoredMinEntries = 1ull << 24;

// The matrix's work area is there, or is allocated now.  Where that fails the
// product that was replaced serves from then on (until cg_spmm_set_format asks
// for the factored form again).  A stored matrix takes the area when it is
// built, an on-the-fly one with its first FP32 product: the path is there for
// problems that fill the device, and a solve's vectors come first.
bool factored_ready(const Hamiltonian& h);
// f(), and where its memory runs out, once more without what products keep
// (that product then stays with the one the factored form replaced).
template <class F>
auto with_room(const Hamiltonian& h, F&& f) {
  try {
    return f();
  } catch (const Error& e) {
    const bool area = h.fact && h.fact->z.p;
    if (e.code != CG_ERR_NOMEM || !h.release_work()) throw;
    h.fact_failed |= area;
    return f();
  }
}

// Y = H X from x packed as n rows of 8 FP32 vectors (32-byte aligned).
// Asynchronous; allocates nothing (factored_ready has been called).
void factored_product_f32(const FactoredOp& f, const float* x, float* y, int ldy, int m, cudaStream_t s);

}  // namespace cg
