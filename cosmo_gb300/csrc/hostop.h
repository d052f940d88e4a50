// Host view of the forward-ordered operator terms: one- and two-body values on
// global occupation words, with the stored builder's fermion phases
// (SM::ActFermiOperator, include/sm/cioperators.cxx:36-62).  Used by the
// host-built tables of the on-the-fly (virtual.cu) and factored (factored.cu)
// products.
#pragma once
#include <cstdint>
#include <vector>

#include "model.h"

namespace cg {

inline int popc(uint64_t x) { return __builtin_popcountll(x); }
inline uint64_t below_h(int b) { return b >= 64 ? ~0ull : (1ull << b) - 1ull; }
// global occupation words (neutron s.p. states from bit 0, protons above) of
// up to 128 s.p. states, host only
using G = unsigned __int128;
inline int popg(G x) { return __builtin_popcountll(uint64_t(x)) + __builtin_popcountll(uint64_t(x >> 64)); }
inline G below_g(int b) { return b >= 128 ? ~G(0) : ((G(1) << b) - 1); }
inline G gbit(int b) { return G(1) << b; }
inline int ctzg(G x) {
  const uint64_t lo = uint64_t(x);
  return lo ? __builtin_ctzll(lo) : 64 + __builtin_ctzll(uint64_t(x >> 64));
}

struct HostOp {
  int ns = 0, np_pairs = 0;
  std::vector<double> e1;      // ns x ns
  std::vector<double> v2;      // npairs x npairs
  std::vector<int32_t> pidx;   // ns x ns
  double V(int a, int b, int c, int d) const {  // a < b, c < d
    return v2[size_t(pidx[a * ns + b]) * np_pairs + pidx[c * ns + d]];
  }
  // forward two-body term (b0 < b1 annihilated, b2 < b3 created) on S0
  double term2(G S0, int b0, int b1, int b2, int b3) const {
    double v = V(b0, b1, b2, b3);
    int p = popg(S0 & below_g(b0)) + popg(S0 & below_g(b1)) - 1;
    G I = S0 & ~(gbit(b0) | gbit(b1));
    p += popg(I & below_g(b2)) + popg(I & below_g(b3));
    return (p & 1) ? -v : v;
  }
  double term1(G S0, int x, int y) const {
    double v = e1[x * ns + y];
    int p = popg(S0 & below_g(x)) + popg((S0 & ~gbit(x)) & below_g(y));
    return (p & 1) ? -v : v;
  }
};

inline HostOp host_operator(const System& sys, const Operator& op) {
  HostOp h;
  const int ns = int(sys.sps.size());
  h.ns = ns;
  h.pidx.assign(ns * ns, -1);
  int np = 0;
  for (int a = 0; a < ns; ++a)
    for (int b = a + 1; b < ns; ++b) h.pidx[a * ns + b] = np++;
  h.np_pairs = np;
  h.e1.assign(ns * ns, 0.0);
  for (auto& kv : op.one) h.e1[kv.first[0] * ns + kv.first[1]] = kv.second;
  h.v2.assign(size_t(std::max(np, 1)) * std::max(np, 1), 0.0);
  for (auto& kv : op.two) {
    const Key4& k = kv.first;
    if (k[0] >= k[1] || k[2] >= k[3]) continue;  // cannot act on a determinant
    h.v2[size_t(h.pidx[k[0] * ns + k[1]]) * np + h.pidx[k[2] * ns + k[3]]] = kv.second;
  }
  return h;
}

}  // namespace cg
