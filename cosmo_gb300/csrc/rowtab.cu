// Rows of a stored H from sorted move tables (rowtab.h).
//
// The elements are those of the general builder (hbuild.cu): same terms, the
// one-particle moves' sums in the same order, same drop rule, so columns and
// values are bit-identical to it.
#include <algorithm>

#include "rowtab.h"

namespace cg {
namespace {

constexpr double kDrop = 1e-14;
constexpr int kMaxNs = 64;

struct Entry {      // list element: target block start or rank, what moves, value
  uint32_t key, info;
  double val;
};
static_assert(sizeof(Entry) == 16, "Entry layout");
// neutron lists: one neutron a -> c: a | c << 6 | slot << 12 | phase << 21, val the
// one-body term and the neutron spectators (slot of an unchanged 2m only);
// two neutrons: kTwo, val the element.  Own-block lists: kDiag; one proton
// b -> d of unchanged 2m: kOne | b | d << 6 | phase << 12; two protons: kTwo.
constexpr uint32_t kTwo = 0x80000000u, kOne = 0x40000000u, kDiag = 0u;

struct Ctx {
  int ns, nn, np, kn, kp, npairs, nblocks, ndm, dm0, m2max, tp;
  uint64_t n, nconf;
  const uint64_t *noff, *binom, *bstart;
  const uint32_t *pcrank, *bmask, *bclass, *cstart, *cmask;
  const double *e1, *v2;
  const int8_t* m2;
};

__device__ __forceinline__ uint32_t below32(int b) { return b >= 32 ? ~0u : (1u << b) - 1u; }
__device__ __forceinline__ int pair_of(const Ctx& c, int a, int b) {  // a < b
  return a * c.ns - a * (a + 1) / 2 + (b - a - 1);
}
__device__ __forceinline__ double v_of(const Ctx& c, int a, int b, int d, int e) {
  return __ldg(c.v2 + size_t(pair_of(c, a, b)) * c.npairs + pair_of(c, d, e));
}
__device__ __forceinline__ uint64_t colex32(uint32_t mask, const uint64_t* binom) {
  uint64_t r = 0;
  for (int i = 1; mask; mask &= mask - 1, ++i) r += binom[(__ffs(mask) - 1) * kBinom + i];
  return r;
}
__device__ __forceinline__ int slot_of(const Ctx& c, int from, int to) {
  return (int(c.m2[to]) - int(c.m2[from])) / 2 + c.m2max;
}
// phase of moving one particle from -> to inside a species mask
__device__ __forceinline__ uint32_t move_phase(uint32_t mask, int from, int to) {
  const uint32_t o = mask & ~(1u << from);
  return uint32_t(__popc(o & below32(from)) + __popc(o & below32(to))) & 1u;
}
// forward two-body term inside one species (local indices, g0 the first global one)
__device__ __forceinline__ double term2(const Ctx& c, int g0, uint32_t S0, int b0, int b1, int b2, int b3) {
  const double v = v_of(c, g0 + b0, g0 + b1, g0 + b2, g0 + b3);
  int p = __popc(S0 & below32(b0)) + __popc(S0 & below32(b1)) - 1;
  const uint32_t I = S0 & ~((1u << b0) | (1u << b1));
  p += __popc(I & below32(b2)) + __popc(I & below32(b3));
  return (p & 1) ? -v : v;
}

// Visit the pairs a < b -> cc < d of one species mask that keep 2m:
// emit(target mask, value of the forward element).
template <class F>
__device__ void two_moves(const Ctx& c, int g0, int norb, uint32_t S, F&& emit) {
  const uint32_t holes = ~S & below32(norb);
  for (uint32_t t = S; t; t &= t - 1) {
    const int a = __ffs(t) - 1;
    for (uint32_t u = t & (t - 1); u; u &= u - 1) {
      const int b = __ffs(u) - 1;
      const int msum = c.m2[g0 + a] + c.m2[g0 + b];
      for (uint32_t w = holes; w; w &= w - 1) {
        const int cc = __ffs(w) - 1;
        for (uint32_t z = w & (w - 1); z; z &= z - 1) {
          const int d = __ffs(z) - 1;
          if (c.m2[g0 + cc] + c.m2[g0 + d] != msum) continue;
          const uint32_t K = S ^ (1u << a) ^ (1u << b) ^ (1u << cc) ^ (1u << d);
          const bool fwd = (a < cc) || (a == cc && b < d);
          emit(K, fwd ? term2(c, g0, S, a, b, cc, d) : term2(c, g0, K, cc, d, a, b));
        }
      }
    }
  }
}

// Neutron list of each block (thread per block): counts, or entries at off[block].
template <bool FILL>
__global__ void k_nlist(Ctx c, uint32_t* __restrict__ cnt, const uint64_t* __restrict__ off, Entry* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.nblocks) return;
  const uint32_t nu = c.bmask[i], holes = ~nu & below32(c.nn);
  uint64_t p = FILL ? off[i] : 0;
  auto emit = [&](uint64_t start, uint32_t info, double val) {
    if (FILL) out[p] = Entry{uint32_t(start), info, val};
    ++p;
  };
  for (uint32_t t = nu; t; t &= t - 1) {
    const int a = __ffs(t) - 1;
    for (uint32_t w = holes; w; w &= w - 1) {
      const int f = __ffs(w) - 1;
      const uint32_t nu2 = nu ^ (1u << a) ^ (1u << f);
      const uint64_t start = c.noff[colex32(nu2, c.binom)];
      if (start == ~0ull) continue;
      const int slot = slot_of(c, a, f);
      double val = 0.0;
      if (FILL && slot == c.dm0) {
        const int x = min(a, f), y = max(a, f);
        const uint32_t S0 = a < f ? nu : nu2;
        const double e = __ldg(c.e1 + x * c.ns + y);
        val = ((__popc(S0 & below32(x)) + __popc((S0 & ~(1u << x)) & below32(y))) & 1) ? -e : e;
        for (uint32_t q = nu & ~(1u << a); q; q &= q - 1) {
          const int sc = __ffs(q) - 1;
          val += term2(c, 0, S0, min(x, sc), max(x, sc), min(y, sc), max(y, sc));
        }
      }
      emit(start, uint32_t(a) | (uint32_t(f) << 6) | (uint32_t(slot) << 12) | (move_phase(nu, a, f) << 21), val);
    }
  }
  two_moves(c, 0, c.nn, nu, [&](uint32_t K, double v) {
    if (fabs(v) >= kDrop) emit(c.noff[colex32(K, c.binom)], kTwo, v);
  });
  if (!FILL) cnt[i] = uint32_t(p);
}

// Own-block list of each proton configuration (thread per configuration).
template <bool FILL>
__global__ void k_olist(Ctx c, uint32_t* __restrict__ cnt, const uint64_t* __restrict__ off, Entry* __restrict__ out) {
  const uint64_t g = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (g >= c.nconf) return;
  const uint32_t pi = c.cmask[g], holes = ~pi & below32(c.np);
  uint64_t p = FILL ? off[g] : 0;
  auto emit = [&](uint32_t rank, uint32_t info, double val) {
    if (FILL) out[p] = Entry{rank, info, val};
    ++p;
  };
  emit(c.pcrank[colex32(pi, c.binom)], kDiag, 0.0);
  for (uint32_t t = pi; t; t &= t - 1) {
    const int b = __ffs(t) - 1;
    for (uint32_t w = holes; w; w &= w - 1) {
      const int d = __ffs(w) - 1;
      if (slot_of(c, c.nn + b, c.nn + d) != c.dm0) continue;
      emit(c.pcrank[colex32(pi ^ (1u << b) ^ (1u << d), c.binom)],
           kOne | uint32_t(b) | (uint32_t(d) << 6) | (move_phase(pi, b, d) << 12), 0.0);
    }
  }
  two_moves(c, c.nn, c.np, pi, [&](uint32_t K, double v) {
    if (fabs(v) >= kDrop) emit(c.pcrank[colex32(K, c.binom)], kTwo, v);
  });
  if (!FILL) cnt[g] = uint32_t(p);
}

// Ascending keys inside every list (a warp each; keys are distinct): every
// element finds its rank among the others.  src and dst differ.
__global__ void k_order(uint64_t nlists, const uint64_t* __restrict__ off, const Entry* __restrict__ src,
                        Entry* __restrict__ dst) {
  const uint64_t i = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= nlists) return;
  const uint64_t b = off[i], e = off[i + 1];
  for (uint64_t p = b + lane; p < e; p += 32) {
    const Entry x = src[p];
    uint32_t r = 0;
    for (uint64_t q = b; q < e; ++q) r += src[q].key < x.key;
    dst[b + r] = x;
  }
}

// One-proton moves of each configuration by slot, then target rank (a warp
// each): pt[g * tp ..] = {rank, b | d << 6 | phase << 12}, poff[g * (ndm + 1) + slot].
__global__ void k_plist(Ctx c, uint2* __restrict__ pt, uint16_t* __restrict__ poff) {
  extern __shared__ uint2 sm[];  // per warp: tp entries {rank, slot << 16 | move}
  const int lane = threadIdx.x & 31;
  uint2* e = sm + (threadIdx.x >> 5) * c.tp;
  const uint64_t g = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  if (g >= c.nconf) return;
  const uint32_t pi = c.cmask[g], holes = ~pi & below32(c.np);
  const int nh = c.np - c.kp;
  for (int i = lane; i < c.tp; i += 32) {
    const int b = __fns(pi, 0, i / nh + 1), d = __fns(holes, 0, i % nh + 1);
    e[i] = make_uint2(c.pcrank[colex32(pi ^ (1u << b) ^ (1u << d), c.binom)],
                      (uint32_t(slot_of(c, c.nn + b, c.nn + d)) << 16) | uint32_t(b) | (uint32_t(d) << 6) |
                          (move_phase(pi, b, d) << 12));
  }
  __syncwarp();
  auto before = [](uint2 x, uint2 y) { return (x.y >> 16) != (y.y >> 16) ? (x.y >> 16) < (y.y >> 16) : x.x < y.x; };
  for (int i = lane; i < c.tp; i += 32) {
    const uint2 x = e[i];
    int r = 0;
    for (int q = 0; q < c.tp; ++q) r += before(e[q], x);
    pt[g * c.tp + r] = make_uint2(x.x, x.y & 0xffffu);
  }
  for (int s = lane; s <= c.ndm; s += 32) {
    int r = 0;
    for (int q = 0; q < c.tp; ++q) r += int(e[q].y >> 16) < s;
    poff[g * (c.ndm + 1) + s] = uint16_t(r);
  }
}

// nz bit (a, c, b, d): the neutron a -> c, proton b -> d element is kept
__global__ void k_nonzero(Ctx c, uint32_t* __restrict__ nz, int words) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.nn * c.nn * words) return;
  const int w = i % words, ac = i / words, a = ac / c.nn, f = ac % c.nn;
  uint32_t m = 0;
  for (int k = 0; k < 32; ++k) {
    const int bd = w * 32 + k;
    if (bd >= c.np * c.np || a == f) break;
    const int b = bd / c.np, d = bd % c.np;
    if (b == d) continue;
    const double v = a < f ? v_of(c, a, c.nn + b, f, c.nn + d) : v_of(c, f, c.nn + d, a, c.nn + b);
    if (fabs(v) >= kDrop) m |= 1u << k;
  }
  nz[i] = m;
}

// diagonal in the general builder's order: one-body terms, then the pairs
__global__ void k_diagonal(Ctx c, const uint64_t* __restrict__ state, double* __restrict__ diag) {
  const uint64_t row = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (row >= c.n) return;
  const uint64_t S = state[row];
  double v = 0.0;
  for (uint64_t t = S; t; t &= t - 1) {
    const int a = __ffsll((long long)t) - 1;
    v += __ldg(c.e1 + a * c.ns + a);
  }
  for (uint64_t t = S; t; t &= t - 1) {
    const int a = __ffsll((long long)t) - 1;
    for (uint64_t u = t & (t - 1); u; u &= u - 1) {
      const int b = __ffsll((long long)u) - 1;
      const int p = pair_of(c, a, b);
      v += __ldg(c.v2 + size_t(p) * c.npairs + p);
    }
  }
  diag[row] = fabs(v) >= kDrop ? v : 0.0;
}

struct Lists {
  const uint64_t *noff, *ooff;  // list starts: neutron blocks, proton configurations
  const Entry *nl, *ol;
  const uint2* pt;
  const uint16_t* poff;
  const uint32_t* nz;
  int words;
};

// one neutron a -> f of unchanged 2m, same protons: the neutron part plus the proton spectators
__device__ __forceinline__ double n1_value(const Ctx& c, const Entry& e, uint32_t pi) {
  const int a = e.info & 63, f = (e.info >> 6) & 63, x = min(a, f), y = max(a, f);
  const bool neg = (e.info >> 21) & 1;
  double v = e.val;
  for (uint32_t w = pi; w; w &= w - 1) {
    const int q = c.nn + __ffs(w) - 1;
    const double t = v_of(c, x, q, y, q);
    v += neg ? -t : t;
  }
  return v;
}
// one proton b -> d of unchanged 2m, same neutrons
__device__ __forceinline__ double p1_value(const Ctx& c, const Entry& e, uint32_t nu, uint32_t pi) {
  const int b = e.info & 63, d = (e.info >> 6) & 63, x = min(b, d), y = max(b, d);
  const bool neg = (e.info >> 12) & 1;
  const double t1 = __ldg(c.e1 + (c.nn + x) * c.ns + c.nn + y);
  double v = neg ? -t1 : t1;
  for (uint32_t w = nu; w; w &= w - 1) {
    const int q = __ffs(w) - 1;
    const double t = v_of(c, q, c.nn + x, q, c.nn + y);
    v += neg ? -t : t;
  }
  const uint32_t S0 = b < d ? pi : pi ^ (1u << b) ^ (1u << d);
  for (uint32_t w = pi & ~(1u << b); w; w &= w - 1) {
    const int sc = __ffs(w) - 1;
    v += term2(c, c.nn, S0, min(x, sc), max(x, sc), min(y, sc), max(y, sc));
  }
  return v;
}

// A warp per row, one lane per list element; the rows of a block share its
// neutron list.  COUNT: elements kept.  Else: the row is laid out in shared
// memory (every list at its full length), compacted and written coalesced.
// fp 3+4, 2.5e8 elements: count 2.0 + fill 5.5 ms (3.0 GB written), where the
// general builder takes 5.0 + 7.2 ms and 8.1 ms to sort the rows; bound by the
// lookups of the two-body table and by lists of unequal length in a warp.
constexpr int kRowsPerWarp = 8;
constexpr size_t kSmemRow = 200 * 1024;  // of a CTA's rows
template <bool COUNT>
__global__ void __launch_bounds__(256) k_rows(Ctx c, Lists l, uint32_t* __restrict__ counts, int cap,
                                              const uint64_t* __restrict__ rowptr, uint32_t* __restrict__ col,
                                              double* __restrict__ out64, float* __restrict__ hi,
                                              float* __restrict__ lo, const double* __restrict__ diag,
                                              unsigned long long* __restrict__ upper,
                                              unsigned* __restrict__ longest) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* sval = reinterpret_cast<double*>(raw) + size_t(warp) * cap;
  uint32_t* scol = reinterpret_cast<uint32_t*>(reinterpret_cast<double*>(raw) + size_t(blockDim.x >> 5) * cap) +
                   size_t(warp) * cap;
  const uint64_t row0 = (blockIdx.x * uint64_t(blockDim.x >> 5) + warp) * kRowsPerWarp;
  if (row0 >= c.n) return;
  int lob = 0, hib = c.nblocks - 1;
  while (lob < hib) {
    const int mid = (lob + hib + 1) >> 1;
    if (c.bstart[mid] <= row0) lob = mid; else hib = mid - 1;
  }
  int beta = lob;
  unsigned up = 0, most = 0;  // entries on or above the diagonal; longest row before the drops
  for (uint64_t row = row0; row < min(c.n, row0 + kRowsPerWarp); ++row) {
    while (beta + 1 < c.nblocks && c.bstart[beta + 1] <= row) ++beta;
    const uint64_t start = c.bstart[beta];
    const uint32_t r = uint32_t(row - start), nu = c.bmask[beta];
    const uint64_t g = c.cstart[c.bclass[beta]] + r;
    const uint32_t pi = c.cmask[g];
    const uint2* pt = l.pt + g * c.tp;
    const uint16_t* po = l.poff + g * (c.ndm + 1);
    const uint64_t n0 = l.noff[beta], n1 = l.noff[beta + 1], o0 = l.ooff[g], o1 = l.ooff[g + 1];
    uint32_t pos = 0, full = uint32_t(o1 - o0);
    bool own_done = false;
    auto own = [&]() {
      for (uint64_t e0 = o0; e0 < o1; e0 += 32) {
        const uint64_t i = e0 + lane;
        double v = 0.0;
        uint32_t key = 0;
        if (i < o1) {
          const Entry e = l.ol[i];
          key = e.key;
          if (e.info & kTwo) v = e.val;
          else if (e.info & kOne) v = p1_value(c, e, nu, pi);
          else v = diag[row];
        }
        if constexpr (COUNT) {
          pos += __popc(__ballot_sync(0xffffffffu, fabs(v) >= kDrop));
        } else {
          if (i < o1) {
            scol[pos + lane] = uint32_t(start) + key;
            sval[pos + lane] = v;
          }
          pos += uint32_t(min(uint64_t(32), o1 - e0));
        }
      }
    };
    for (uint64_t e0 = n0; e0 < n1 || !own_done; e0 += 32) {
      // lists of the targets below the own block come first
      const uint64_t i = e0 + lane;
      Entry e{~0u, kTwo, 0.0};
      if (i < n1) e = l.nl[i];
      const uint32_t low = __ballot_sync(0xffffffffu, i < n1 && e.key < uint32_t(start));
      uint32_t len = 0, p0 = 0, p1 = 0;
      bool flat = false;
      if (i < n1) {
        if (e.info & kTwo) {
          len = 1;
        } else {
          const int slot = (e.info >> 12) & 0x1ff;
          p0 = po[2 * c.m2max - slot];
          p1 = po[2 * c.m2max - slot + 1];
          flat = slot == c.dm0;
          len = p1 - p0 + flat;
        }
      }
      if constexpr (COUNT) {
        uint32_t k = 0;
        if (i < n1) {
          if (e.info & kTwo) {
            k = 1;
          } else {
            const uint32_t* nz = l.nz + ((e.info & 63) * c.nn + ((e.info >> 6) & 63)) * l.words;
            for (uint32_t p = p0; p < p1; ++p) {
              const uint32_t mv = pt[p].y, bd = (mv & 63) * c.np + ((mv >> 6) & 63);
              k += (nz[bd >> 5] >> (bd & 31)) & 1u;
            }
            if (flat) k += fabs(n1_value(c, e, pi)) >= kDrop;
          }
        }
        pos += __reduce_add_sync(0xffffffffu, k);
        full += __reduce_add_sync(0xffffffffu, len);
        if (!own_done && low != 0xffffffffu) {
          own();
          own_done = true;
        }
      } else {
        uint32_t inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += t;
        }
        // the own block's list goes between the lists below and above it
        const bool here = !own_done && low != 0xffffffffu;
        const int nlow = here ? __popc(low) : 32;
        uint32_t base = pos + inc - len;
        const uint32_t below_total = here ? (nlow ? __shfl_sync(0xffffffffu, inc, nlow - 1) : 0u) : 0u;
        if (here) {
          const uint32_t keep = pos;
          pos = keep + below_total;
          own();
          const uint32_t olen = pos - keep - below_total;
          if (lane >= nlow) base += olen;
          pos = keep + olen;
          own_done = true;
        }
        if (i < n1) {
          if (e.info & kTwo) {
            scol[base] = e.key + r;
            sval[base] = e.val;
          } else {
            const int a = e.info & 63, f = (e.info >> 6) & 63;
            const uint32_t neg = (e.info >> 21) & 1u;
            bool todo = flat;
            for (uint32_t p = p0; p < p1; ++p) {
              const uint2 m = pt[p];
              if (todo && m.x > r) {
                scol[base] = e.key + r;
                sval[base++] = n1_value(c, e, pi);
                todo = false;
              }
              const int b = c.nn + int(m.y & 63), d = c.nn + int((m.y >> 6) & 63);
              const double v = a < f ? v_of(c, a, b, f, d) : v_of(c, f, d, a, b);
              scol[base] = e.key + m.x;
              sval[base++] = ((m.y >> 12) ^ neg) & 1u ? -v : v;
            }
            if (todo) {
              scol[base] = e.key + r;
              sval[base] = n1_value(c, e, pi);
            }
          }
        }
        pos += __shfl_sync(0xffffffffu, inc, 31);
      }
    }
    if constexpr (COUNT) {
      if (lane == 0) counts[row] = pos;
      most = max(most, full);
    } else {
      __syncwarp();
      uint64_t w = rowptr[row];
      for (uint32_t i0 = 0; i0 < pos; i0 += 32) {
        const uint32_t i = i0 + lane;
        const double v = i < pos ? sval[i] : 0.0;
        const bool keep = fabs(v) >= kDrop;
        const uint32_t m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const uint64_t q = w + __popc(m & ((1u << lane) - 1u));
          const uint32_t cc = scol[i];
          col[q] = cc;
          if (out64) out64[q] = v;
          if (hi) {
            const float h = float(v);
            hi[q] = h;
            lo[q] = float(v - double(h));
          }
          up += cc >= row;
        }
        w += __popc(m);
      }
      __syncwarp();
    }
  }
  if constexpr (COUNT) {
    if (lane == 0) atomicMax(longest, most);
  } else {
    up = __reduce_add_sync(0xffffffffu, up);
    if (lane == 0 && up) atomicAdd(upper, (unsigned long long)up);
  }
}

struct Impl : RowTables {
  Ctx c{};
  Lists l{};
  const uint64_t* state = nullptr;
  cudaStream_t s = nullptr;
  DBuf<uint64_t> bstart, noff, ooff;
  DBuf<uint32_t> bmask, bclass, cstart, cmask, nz;
  DBuf<int8_t> m2;
  DBuf<Entry> nl, ol;
  DBuf<uint2> pt;
  DBuf<uint16_t> poff;
  DBuf<double> diag;
  DBuf<unsigned> longest;
  int cap = 0;  // longest row before the drops (after count)

  // list starts from counts (host scan); uses += entries x rows that read them
  template <class W>
  uint64_t starts(const DBuf<uint32_t>& cnt, uint64_t k, DBuf<uint64_t>& off, W&& rows, uint64_t& uses) {
    std::vector<uint32_t> h(k);
    CG_CUDA(cudaMemcpyAsync(h.data(), cnt.p, k * 4, cudaMemcpyDeviceToHost, s));
    CG_CUDA(cudaStreamSynchronize(s));
    std::vector<uint64_t> o(k + 1, 0);
    for (uint64_t i = 0; i < k; ++i) {
      o[i + 1] = o[i] + h[i];
      uses += h[i] * rows(i);
    }
    off.upload(o, s);
    CG_CUDA(cudaStreamSynchronize(s));  // o leaves
    return o[k];
  }
  template <class G>
  void lists(uint64_t k, uint64_t total, const DBuf<uint64_t>& off, DBuf<Entry>& out, G&& fill) {
    DBuf<Entry> raw(std::max<uint64_t>(total, 1));
    out.alloc(std::max<uint64_t>(total, 1));
    fill(off.p, raw.p);
    CG_CUDA(cudaGetLastError());
    k_order<<<unsigned((k * 32 + 255) / 256), 256, 0, s>>>(k, off.p, raw.p, out.p);
    CG_CUDA(cudaGetLastError());
    count_launch(2);
    CG_CUDA(cudaStreamSynchronize(s));  // raw leaves
  }

  size_t smem() const { return size_t(8) * cap * 12; }
  unsigned grid() const { return unsigned((c.n + 8 * kRowsPerWarp - 1) / (8 * kRowsPerWarp)); }
  bool count(uint32_t* counts) override {
    CG_CUDA(cudaMemsetAsync(longest.p, 0, sizeof(unsigned), s));
    k_rows<true><<<grid(), 256, 0, s>>>(c, l, counts, 0, nullptr, nullptr, nullptr, nullptr, nullptr, diag.p, nullptr,
                                        longest.p);
    CG_CUDA(cudaGetLastError());
    count_launch();
    unsigned m = 0;
    CG_CUDA(cudaMemcpyAsync(&m, longest.p, sizeof(m), cudaMemcpyDeviceToHost, s));
    CG_CUDA(cudaStreamSynchronize(s));
    cap = int((m + 1) & ~1u);
    return smem() <= kSmemRow;
  }
  void fill(const uint64_t* rowptr, uint32_t* col, double* out64, float* hi, float* lo, double* dg,
            unsigned long long* upper) override {
    CG_CUDA(cudaFuncSetAttribute(k_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    k_rows<false><<<grid(), 256, smem(), s>>>(c, l, nullptr, cap, rowptr, col, out64, hi, lo, diag.p, upper, nullptr);
    CG_CUDA(cudaGetLastError());
    count_launch();
    CG_CUDA(cudaMemcpyAsync(dg, diag.p, c.n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  }
};

std::unique_ptr<RowTables> make_tables(const Basis& b, const DevOperator& op, cudaStream_t s) {
  if (b.wide || b.truncated || !b.n || b.n >= (1ull << 32) || b.ns > kMaxNs) return nullptr;
  // one parity per species and half-integer (or integer) 2m throughout: the
  // change of 2m alone then pairs neutron and proton moves
  for (int i = 0; i < b.ns; ++i) {
    const int ref = i < b.nn ? 0 : b.nn;
    if (b.sp_par[i] != b.sp_par[ref] || ((b.sp_m2[i] - b.sp_m2[0]) & 1)) return nullptr;
  }
  auto t = std::make_unique<Impl>();
  Ctx& c = t->c;
  t->s = s;
  c.ns = b.ns;
  c.nn = b.nn;
  c.np = b.np;
  c.kn = b.kn;
  c.kp = b.kp;
  c.npairs = op.npairs;
  c.n = b.n;
  c.nblocks = int(b.h_bstart.size());
  // the proton configurations of the classes that some block uses, class by class
  const size_t nclass = b.h_cstart.size();
  const auto class_end = [&](size_t i) { return i + 1 < nclass ? b.h_cstart[i + 1] : uint32_t(b.h_cmasks.size()); };
  std::vector<uint64_t> blocks(nclass, 0);  // of each class
  for (uint32_t k : b.h_bclass) ++blocks[k];
  std::vector<uint32_t> cstart(nclass, 0), cmask, of;
  for (size_t i = 0; i < nclass; ++i) {
    cstart[i] = uint32_t(cmask.size());
    if (!blocks[i]) continue;
    cmask.insert(cmask.end(), b.h_cmasks.begin() + b.h_cstart[i], b.h_cmasks.begin() + class_end(i));
    of.resize(cmask.size(), uint32_t(i));
  }
  c.nconf = cmask.size();
  for (int i = 0; i < b.ns; ++i) c.m2max = std::max(c.m2max, std::abs(b.sp_m2[i]));
  c.ndm = 2 * c.m2max + 1;
  c.dm0 = c.m2max;
  c.tp = c.kp * (c.np - c.kp);
  if (c.ndm > 0x1ff || size_t(c.tp) * 8 * sizeof(uint2) > 48 * 1024) return nullptr;
  t->bstart.upload(b.h_bstart, s);
  t->bmask.upload(b.h_bmask, s);
  t->bclass.upload(b.h_bclass, s);
  t->cstart.upload(cstart, s);
  t->cmask.upload(cmask, s);
  std::vector<int8_t> m2(b.sp_m2.begin(), b.sp_m2.end());
  t->m2.upload(m2, s);
  c.noff = b.noff.p;
  c.binom = b.binom.p;
  c.pcrank = b.pcrank.p;
  c.e1 = op.e1.p;
  c.v2 = op.v2.p;
  c.bstart = t->bstart.p;
  c.bmask = t->bmask.p;
  c.bclass = t->bclass.p;
  c.cstart = t->cstart.p;
  c.cmask = t->cmask.p;
  c.m2 = t->m2.p;
  const unsigned gb = unsigned((c.nblocks + 63) / 64), gc = unsigned((c.nconf + 63) / 64);
  DBuf<uint32_t> ncnt(std::max(c.nblocks, 1)), ocnt(std::max<uint64_t>(c.nconf, 1));
  k_nlist<false><<<gb, 64, 0, s>>>(c, ncnt.p, nullptr, nullptr);
  CG_CUDA(cudaGetLastError());
  k_olist<false><<<gc, 64, 0, s>>>(c, ocnt.p, nullptr, nullptr);
  CG_CUDA(cudaGetLastError());
  count_launch(2);
  uint64_t uses = 0;
  const uint64_t nls = t->starts(ncnt, c.nblocks, t->noff,
                                 [&](uint64_t i) { return uint64_t(class_end(b.h_bclass[i])) - b.h_cstart[b.h_bclass[i]]; },
                                 uses);
  const uint64_t ols = t->starts(ocnt, c.nconf, t->ooff, [&](uint64_t g) { return blocks[of[g]]; }, uses);
  const uint64_t moves = c.kn ? c.nconf * (c.tp * sizeof(uint2) + (c.ndm + 1) * sizeof(uint16_t)) : 0;
  if (!row_tables_worth((nls + ols) * 2 * sizeof(Entry) + moves, uses)) return nullptr;
  t->lists(c.nblocks, nls, t->noff, t->nl,
           [&](const uint64_t* o, Entry* e) { k_nlist<true><<<gb, 64, 0, s>>>(c, nullptr, o, e); });
  t->lists(c.nconf, ols, t->ooff, t->ol,
           [&](const uint64_t* o, Entry* e) { k_olist<true><<<gc, 64, 0, s>>>(c, nullptr, o, e); });
  if (c.kn) {  // else no neutron moves, and nothing reads them
    t->pt.alloc(std::max<uint64_t>(c.nconf * c.tp, 1));
    t->poff.alloc(c.nconf * (c.ndm + 1));
    k_plist<<<unsigned((c.nconf * 32 + 255) / 256), 256, size_t(c.tp) * 8 * sizeof(uint2), s>>>(c, t->pt.p, t->poff.p);
    CG_CUDA(cudaGetLastError());
    count_launch();
  }
  const int words = (c.np * c.np + 31) / 32;
  t->nz.alloc(std::max(c.nn * c.nn * words, 1));
  if (c.nn && c.np) {
    k_nonzero<<<unsigned((c.nn * c.nn * words + 127) / 128), 128, 0, s>>>(c, t->nz.p, words);
    CG_CUDA(cudaGetLastError());
    count_launch();
  }
  t->diag.alloc(c.n);
  k_diagonal<<<unsigned((c.n + 255) / 256), 256, 0, s>>>(c, b.state.p, t->diag.p);
  CG_CUDA(cudaGetLastError());
  count_launch();
  t->longest.alloc(1);
  t->l = Lists{t->noff.p, t->ooff.p, t->nl.p, t->ol.p, t->pt.p, t->poff.p, t->nz.p, words};
  return t;
}

}  // namespace

std::unique_ptr<RowTables> row_tables(const Basis& b, const DevOperator& op, cudaStream_t s) {
  try {
    return make_tables(b, op, s);
  } catch (const Error& e) {
    if (e.code != CG_ERR_NOMEM) throw;
    return nullptr;  // what was allocated is free again; the general builder needs no tables
  }
}

}  // namespace cg
