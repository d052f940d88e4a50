// Factored H + lambda * J-J+ product (the decomposition is in factored.h).
//
// k_fact32: one CTA per (core, spectator group): the channel's matrix goes to
// shared memory once, the spectators' rows of x are gathered chunk by chunk,
// and every warp forms 16 x 16 output rows of 8 vectors in registers.
// k_pair32: the same for two particles of one species, whose rows fit in
// registers.  Every (slot, row) of the work area is written by exactly one
// thread, where the slot numbers the pair of particles of the row that the
// core lacks, so the partial sums need no atomics and k_fsum adds them in a
// fixed order: the product is deterministic.
#include <algorithm>
#include <cmath>
#include <map>

#include "factored.h"
#include "hostop.h"

namespace cg {
namespace {

constexpr int kFMaxPairs = 128;  // pairs of a channel
constexpr int kFSmem = 56 * 1024;
constexpr double kFDrop = 1e-14;  // smaller elements are zeros, as in a stored matrix

struct FArgs {
  uint64_t n;
  int cols;  // states of the spectators' species
  const FJob* jobs;
  const FPair* list;
  const uint32_t *stab, *spect;
};

__device__ __forceinline__ int meta_idx(uint32_t m) { return int(m & 0xffu); }
__device__ __forceinline__ int meta_b(uint32_t m) { return int((m >> 8) & 0xffu); }
__device__ __forceinline__ uint32_t meta_slot(uint32_t m) { return (m >> 16) & 0x7fffu; }
// A spectator's table entry: for neutron + proton pairs the row offset and,
// from bit 27, the position of the particle (its parity is the spectator's
// phase); for pairs of one species the row offset alone.
constexpr int kFPosBit = 27;
constexpr uint32_t kFOff = (1u << kFPosBit) - 1u;
__device__ __forceinline__ uint32_t pos_phase(uint32_t o) { return (o << (31 - kFPosBit)) & 0x80000000u; }

struct Row32 {
  uint32_t v[8];
};
__device__ __forceinline__ void st_row(void* p, const Row32& r) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r.v[0]), "r"(r.v[1]), "r"(r.v[2]),
               "r"(r.v[3]), "r"(r.v[4]), "r"(r.v[5]), "r"(r.v[6]), "r"(r.v[7])
               : "memory");
}

__device__ __forceinline__ void fma2(float2& c, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(c))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid = true) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
// every cp.async of the thread, committed or not
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// FP32 product of 8 vectors, neutron + proton pairs.  Bound by the FP32 pipe in
// principle (fp 4 + 4: 1.7e9 multiply-adds x 8 with filled-up tiles, 0.35 ms); it
// takes 0.85 ms, the rest waiting at the two barriers of a chunk.  Four warps a
// CTA and four CTAs an SM measured best (3, 5, 6, 8 warps with tiles of 8: 1.00,
// 0.91, 0.98, 1.10 ms against 0.89; rows fetched in two alternating halves 0.90).
// A warp forms tiles of 2 groups of OT <= 8 outputs x 16 spectators (fact_tiles).
// The lane's bit 1 picks the group and the other bits the spectator: lanes i and
// i ^ 1 read the same piece of the matrix and lanes i and i ^ 2 the same piece of
// x, so that every 16-byte shared-memory read of the warp takes two cycles
// instead of four.
constexpr int kFW = 4;  // warps

// shared-memory head of the FP32 kernels: the pairs of the job
struct alignas(16) FHead32 {
  uint2 src[kFMaxPairs];    // first row of block core + a; b
  uint64_t dst[kFMaxPairs]; // first row in the work area: slot n + src
  uint32_t meta[kFMaxPairs];
};

// Infinities and NaN.  The channel's matrix is dense, so a row of x that is not
// finite would turn every output of its cores into NaN through the zeros of the
// matrix, where the element-wise products reach connected rows only.  It shows
// in any one output: where that is not finite, all are formed again without the
// zeros (an infinity still comes out as NaN where the terms of an element differ
// in sign).  fp 4 + 4: 1.367 -> 1.377 ms a product.
template <int N>
__device__ __forceinline__ bool not_finite(const float2 (&v)[N]) {
  float2 c = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < N; ++i) fma2(c, v[i], make_float2(0.f, 0.f));
  return !(c.x + c.y == 0.f);
}

// Output o of a tile's spectator once more, without the zeros of its matrix column wp
__device__ __noinline__ void redo_row(const FArgs& a, const FHead32& hd, int o, int D, const float* wp, int wld,
                                      const float4* xp, const uint32_t* sp, int ld, const uint32_t* of,
                                      unsigned char* z) {
  const uint32_t at = of[hd.src[o].y];
  if (at == ~0u) return;
  float2 acc[4] = {};
  for (int k = 0; k < D; ++k) {
    const float w = __uint_as_float(__float_as_uint(wp[k * wld]) ^ sp[k * ld]);
    if (w == 0.f) continue;
    const float4 x0 = xp[2 * ld * k], x1 = xp[2 * ld * k + ld];
    const float2 w2 = make_float2(w, w), xv[4] = {{x0.x, x0.y}, {x0.z, x0.w}, {x1.x, x1.y}, {x1.z, x1.w}};
    for (int v = 0; v < 4; ++v) fma2(acc[v], w2, xv[v]);
  }
  const uint64_t row = hd.dst[o] + (at & kFOff) + uint64_t(at >> kFPosBit) * a.n;
  Row32 r;
  for (int v = 0; v < 4; ++v) {
    r.v[2 * v] = __float_as_uint(acc[v].x) ^ pos_phase(at);
    r.v[2 * v + 1] = __float_as_uint(acc[v].y) ^ pos_phase(at);
  }
  st_row(z + row * 32, r);
}

// One warp tile: acc += matrix rows x gathered rows, then the output rows.  sg
// holds the spectator's phase of each (pair, spectator) as a sign bit, applied
// to the matrix values while they are doubled for the packed multiply-adds.
// A group's OT values lie in 8 places, so that two 16-byte reads fetch them.
template <int OT>
__device__ __forceinline__ void tile32(const FArgs& a, const FHead32& hd, int D, int tile, int j, bool live,
                                       const float* ws, int wld, const float4* xs, const uint32_t* sg, int ld,
                                       const uint32_t* of, unsigned char* __restrict__ z) {
  const int group = tile * 2 + ((threadIdx.x >> 1) & 1);
  float2 acc[OT][4];
#pragma unroll
  for (int t = 0; t < OT; ++t)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[t][v] = make_float2(0.f, 0.f);
  const float* wp = ws + group * 8;
  const float4* xp = xs + j;
  const uint32_t* sp = sg + j;
#pragma unroll 2
  for (int k = 0; k < D; ++k) {
    const float4 x0 = xp[0], x1 = xp[ld];
    const uint32_t f = *sp;
    const float2 xv[4] = {{x0.x, x0.y}, {x0.z, x0.w}, {x1.x, x1.y}, {x1.z, x1.w}};
    const float4 w0 = reinterpret_cast<const float4*>(wp)[0];
    const float4 w1 = OT > 4 ? reinterpret_cast<const float4*>(wp)[1] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int t = 0; t < OT; ++t) {
      const float ws1 = __uint_as_float(__float_as_uint(wv[t]) ^ f);
      const float2 w2 = make_float2(ws1, ws1);
#pragma unroll
      for (int v = 0; v < 4; ++v) fma2(acc[t][v], w2, xv[v]);
    }
    wp += wld;
    xp += 2 * ld;
    sp += ld;
  }
  if (!live) return;
  const bool bad = not_finite(acc[0]);
#pragma unroll
  for (int t = 0; t < OT; ++t) {
    const int k = group * OT + t;
    if (k < D) {
      const uint32_t o = of[hd.src[k].y];
      if (o != ~0u) {
        const uint64_t row = hd.dst[k] + (o & kFOff) + uint64_t(o >> kFPosBit) * a.n;
        const uint32_t f = pos_phase(o);
        Row32 r;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          r.v[2 * v] = __float_as_uint(acc[t][v].x) ^ f;
          r.v[2 * v + 1] = __float_as_uint(acc[t][v].y) ^ f;
        }
        st_row(z + row * 32, r);
      }
    }
  }
  if (bad)
    for (int t = 0; t < OT && group * OT + t < D; ++t)
      redo_row(a, hd, group * OT + t, D, ws + group * 8 + t, wld, xs + j, sg + j, ld, of, z);
}

// Outputs of a job in 1, 2 or 4 warp tiles (more above 64 pairs) of 2 groups of
// OT, as even as they can be: with tiles of 16 one of the four warps was idle
// for 33 to 48 pairs, half of the work of fp 4 + 4 (0.89 ms; so 0.84).
__host__ __device__ inline int fact_tiles(int D) { return D <= 16 ? 1 : D <= 32 ? 2 : D <= 64 ? 4 : (D + 15) / 16; }

__global__ void __launch_bounds__(kFW * 32, 4) k_fact32(FArgs a, const float* __restrict__ w,
                                                        const unsigned char* __restrict__ x,
                                                        unsigned char* __restrict__ z, int smem) {
  constexpr int NT = kFW * 32;
  extern __shared__ __align__(16) unsigned char sm[];
  FHead32& hd = *reinterpret_cast<FHead32*>(sm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const FJob job = a.jobs[blockIdx.x];
  const int count = int(job.count), cols = a.cols, D = int(job.npair);
  const int ot = fact_tiles(D), OT = (D + 2 * ot - 1) / (2 * ot), wld = ot * 16;
  // spectators of a chunk: as many groups of 16 as fill the warps, within the shared memory
  const int cap = (smem - int(sizeof(FHead32)) - D * wld * 4) / (D * 36 + 2 * cols * 4) >> 4;
  const int NK = min(min(max(kFW / ot, 1), cap), (count + 15) >> 4) * 16;
  float* ws = reinterpret_cast<float*>(sm + sizeof(FHead32));
  float4* xs = reinterpret_cast<float4*>(ws + D * wld);
  uint32_t* sg = reinterpret_cast<uint32_t*>(xs + D * NK * 2);
  uint32_t* tab = sg + D * NK;  // two chunks of the spectators' table
  const uint32_t* stab = a.stab + size_t(job.spect) * cols;
  for (int i = tid; i < min(NK, count) * cols; i += NT) cp_async4(tab + i, stab + i);
  for (int k = tid; k < D; k += NT) {
    const FPair p = a.list[job.list + k];
    hd.src[k] = make_uint2(p.row, meta_b(p.meta));
    hd.dst[k] = meta_slot(p.meta) * a.n + p.row;
    hd.meta[k] = p.meta;
  }
  __syncthreads();
  // the matrix restricted to the job's pairs, phases of both sides folded in; a warp per row
  for (int i = lane; i < wld; i += 32) {
    const int o = (i >> 3) * OT + (i & 7);
    const bool used = (i & 7) < OT && o < D;
    const uint32_t mo = used ? hd.meta[o] : 0;
    const float* src = w + job.w0 + meta_idx(mo);
#pragma unroll 8
    for (int k = warp; k < D; k += kFW) {
      const uint32_t mk = hd.meta[k];
      const float v = used ? __ldg(src + meta_idx(mk) * job.ldw) : 0.f;
      ws[k * wld + i] = __uint_as_float(__float_as_uint(v) ^ ((mk ^ mo) & 0x80000000u));
    }
  }
  cp_async_wait_all();
  const int h = tid & 1, q = tid >> 1, jl = (lane & 1) | ((lane >> 2) << 1);
  const unsigned char* xh = x + h * 16;
  uint32_t* cur = tab;
  uint32_t* nxt = tab + NK * cols;
  for (int c0 = 0; c0 < count; c0 += NK) {
    const int cnt = min(NK, count - c0);
    __syncthreads();  // the table has landed; the previous rows are done with
    for (int j = q & 15; j < cnt; j += 16) {
      const uint32_t* of = cur + j * cols;
      float4* xd = xs + h * NK + j + (q >> 4) * 2 * NK;
      uint32_t* sd = sg + j + (q >> 4) * NK;
#pragma unroll 4
      for (int k = q >> 4; k < D; k += kFW) {
        const uint2 p = hd.src[k];
        const uint32_t o = of[p.y];
        const bool ok = o != ~0u;
        cp_async16(xd, xh + uint64_t(p.x + (ok ? o & kFOff : 0u)) * 32, ok);
        if (h == 0) *sd = pos_phase(o);
        xd += kFW * 2 * NK;
        sd += kFW * NK;
      }
    }
    const int left = min(NK, count - c0 - NK) * cols;
    stab += NK * cols;
    for (int i = tid; i < left; i += NT) cp_async4(nxt + i, stab + i);
    cp_async_wait_all();
    __syncthreads();
    const int tiles = ot * ((cnt + 15) >> 4);
    for (int t = warp; t < tiles; t += kFW) {
      const int jt = t / ot, j = jt * 16 + jl, tile = t - jt * ot;
#define CG_TILE(N) tile32<N>(a, hd, D, tile, j, j < cnt, ws, wld, xs, sg, NK, cur + j * cols, z)
      switch (OT) {
        case 8: CG_TILE(8); break;
        case 7: CG_TILE(7); break;
        case 6: CG_TILE(6); break;
        case 5: CG_TILE(5); break;
        case 4: CG_TILE(4); break;
        case 3: CG_TILE(3); break;
        case 2: CG_TILE(2); break;
        default: CG_TILE(1); break;
      }
#undef CG_TILE
    }
    uint32_t* t = cur;
    cur = nxt;
    nxt = t;
  }
}

// FP32 product of 8 vectors, pairs of one species: a thread keeps one 16-byte
// half of its spectator's rows in registers and forms the outputs one after
// another, so nothing but the matrix (phases folded in) is staged.
constexpr int kFPairs = 32;  // pairs of a one-species job

// a spectator's outputs once more (16-byte halves of the rows), without the zeros of the matrix
__device__ __noinline__ void redo_half(int D, const uint32_t* src, const uint64_t* dst, const float* ws,
                                       const unsigned char* x, unsigned char* z, uint32_t off) {
  for (int o = 0; o < D; ++o) {
    float2 acc[2] = {};
    for (int k = 0; k < D; ++k) {
      const float w = ws[o * kFPairs + k];
      if (w == 0.f) continue;
      const float4 r = __ldg(reinterpret_cast<const float4*>(x + uint64_t(src[k] + off) * 32));
      fma2(acc[0], make_float2(w, w), make_float2(r.x, r.y));
      fma2(acc[1], make_float2(w, w), make_float2(r.z, r.w));
    }
    *reinterpret_cast<float4*>(z + (dst[o] + off) * 32) = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
  }
}

template <int DM>
__device__ __forceinline__ void pairs32(const FArgs& a, const FJob& job, int D, const uint32_t* src,
                                        const uint64_t* dst, const float* ws, const unsigned char* __restrict__ x,
                                        unsigned char* __restrict__ z) {
  const int h = threadIdx.x & 1;
  for (uint32_t j = threadIdx.x >> 1; j < job.count; j += 64) {
    const uint32_t off = job.spect == ~0u ? job.first + j : __ldg(a.spect + job.spect + j);
    float2 xv[DM][2];
#pragma unroll
    for (int k = 0; k < DM; ++k) {
      float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < D) r = __ldg(reinterpret_cast<const float4*>(x + uint64_t(src[k] + off) * 32) + h);
      xv[k][0] = make_float2(r.x, r.y);
      xv[k][1] = make_float2(r.z, r.w);
    }
    bool bad = false;
#pragma unroll 2
    for (int o = 0; o < D; ++o) {
      const float4* wp = reinterpret_cast<const float4*>(ws + o * kFPairs);
      float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int k = 0; k < DM; k += 4) {
        const float4 t = wp[k >> 2];
        const float wv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          fma2(acc[0], make_float2(wv[u], wv[u]), xv[k + u][0]);
          fma2(acc[1], make_float2(wv[u], wv[u]), xv[k + u][1]);
        }
      }
      if (o == 0) bad = not_finite(acc);
      reinterpret_cast<float4*>(z + (dst[o] + off) * 32)[h] =
          make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
    }
    if (bad) redo_half(D, src, dst, ws, x + h * 16, z + h * 16, off);
  }
}

__global__ void __launch_bounds__(128) k_pair32(FArgs a, const float* __restrict__ w,
                                                const unsigned char* __restrict__ x, unsigned char* __restrict__ z) {
  __shared__ __align__(16) float ws[kFPairs * kFPairs];  // output-major
  __shared__ uint32_t src[kFPairs], meta[kFPairs];
  __shared__ uint64_t dst[kFPairs];
  const int tid = threadIdx.x;
  const FJob job = a.jobs[blockIdx.x];
  const int D = int(job.npair);
  if (tid < D) {
    const FPair p = a.list[job.list + tid];
    src[tid] = p.row;
    meta[tid] = p.meta;
    dst[tid] = meta_slot(p.meta) * a.n + p.row;
  }
  __syncthreads();
  for (int i = tid; i < D * kFPairs; i += 128) {
    const int o = i / kFPairs, k = i % kFPairs;
    float v = 0.f;
    if (k < D) {
      v = __ldg(w + job.w0 + meta_idx(meta[k]) * job.ldw + meta_idx(meta[o]));
      v = __uint_as_float(__float_as_uint(v) ^ ((meta[k] ^ meta[o]) & 0x80000000u));
    }
    ws[i] = v;
  }
  __syncthreads();
  if (D <= 8) pairs32<8>(a, job, D, src, dst, ws, x, z);
  else if (D <= 16) pairs32<16>(a, job, D, src, dst, ws, x, z);
  else if (D <= 24) pairs32<24>(a, job, D, src, dst, ws, x, z);
  else pairs32<32>(a, job, D, src, dst, ws, x, z);
}

// y[row] = the sum of the row's partial sums, in slot order (vec: y takes
// 16-byte stores and all 8 vectors are wanted).  Reads at the HBM rate (fp
// 4 + 4: 1.76 GB in 0.26 ms).
__global__ void __launch_bounds__(256) k_fsum(uint64_t n, int slots, const float4* __restrict__ z,
                                              float* __restrict__ y, int ldy, int m, bool vec) {
  const uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i >= 2 * n) return;
  const int half = int(i & 1);
  const float4* zp = z + i;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int q = 0; q < slots; ++q) {
    const float4 v = __ldcs(zp + uint64_t(q) * 2 * n);
    s.x += v.x;
    s.y += v.y;
    s.z += v.z;
    s.w += v.w;
  }
  float* yr = y + (i >> 1) * ldy + half * 4;
  if (vec) {
    *reinterpret_cast<float4*>(yr) = s;
  } else {
    const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (half * 4 + j < m) yr[j] = v[j];
  }
}

// masks of k particles in norb states, grouped by (2m, parity): masks in group
// order, and the group starts by key
struct Cores {
  std::vector<uint32_t> mask;
  std::map<std::pair<int, int>, std::pair<uint32_t, uint32_t>> group;  // first, count
};
Cores make_cores(int norb, int k, const int* m2, const int* par) {
  std::map<std::pair<int, int>, std::vector<uint32_t>> by;
  auto add = [&](uint32_t m) {
    int s = 0, p = 0;
    for (uint32_t t = m; t; t &= t - 1) {
      s += m2[__builtin_ctz(t)];
      p ^= par[__builtin_ctz(t)];
    }
    by[{s, p}].push_back(m);
  };
  if (k == 0) {
    add(0);
  } else {
    for (uint64_t m = (1ull << k) - 1, end = 1ull << norb; m < end;) {
      add(uint32_t(m));
      const uint64_t c = m & (~m + 1), r = m + c;
      m = (((r ^ m) >> 2) / c) | r;
    }
  }
  Cores out;
  for (auto& kv : by) {
    out.group[kv.first] = {uint32_t(out.mask.size()), uint32_t(kv.second.size())};
    out.mask.insert(out.mask.end(), kv.second.begin(), kv.second.end());
  }
  return out;
}

std::shared_ptr<FactoredOp> build_tables(const System& sys, const Operator& op, const Basis& b, double other_us,
                                         cudaStream_t s) {
  const int nn = b.nn, np = b.np, ns = b.ns, kn = b.kn, kp = b.kp;
  if (b.wide || b.truncated || !b.n || kn < 1 || kp < 1 || nn > 32 || np > 32) return nullptr;
  const int slots = kn * kp + kn * (kn - 1) / 2 + kp * (kp - 1) / 2;
  if (b.n > kFOff || std::max(kn, kp) > 31 || slots > 0x7fff || slots * 32 * b.n > kFactoredMaxWork) return nullptr;
  // share of a core's pairs that are free: below a half the blocked ones cost
  // more than the cores save (sd 5+5, 0.44: 90 against 93 us; sd 4+4, 0.56: 33 against 65)
  if (double(nn - kn + 1) * (np - kp + 1) < 0.5 * nn * np) return nullptr;
  auto choose = [&](int n, int k) { return k < 0 ? 0 : b.h_binom[n * kBinom + k]; };
  if (choose(nn, kn - 1) > (1u << 22) || choose(np, kp - 1) > (1u << 22)) return nullptr;
  const HostOp H = host_operator(sys, op);
  auto fp = std::make_shared<FactoredOp>();
  FactoredOp& f = *fp;
  f.n = b.n;
  f.slots = slots;
  const int *m2 = b.sp_m2.data(), *par = b.sp_par.data();
  std::vector<uint32_t> bof(std::max<uint64_t>(b.neut.nconf, 1), ~0u);  // block of a neutron configuration
  const int nblocks = int(b.h_bstart.size());
  for (int i = 0; i < nblocks; ++i) bof[colex_host(b.h_bmask[i], b.h_binom)] = uint32_t(i);
  auto start_of = [&](uint32_t m) {
    const uint32_t i = bof[colex_host(m, b.h_binom)];
    return i == ~0u ? ~0u : uint32_t(b.h_bstart[i]);
  };

  struct Chan {
    std::vector<uint16_t> pairs;  // x | y << 8, s.p. states of their species
    uint32_t w0;                  // first value of the matrix
  };
  std::vector<double> w;
  std::vector<FJob> jobs;
  std::vector<FPair> list;
  auto add_job = [&](uint32_t l0, uint32_t spect, uint32_t count, const Chan& c, uint32_t kind) {
    const uint32_t D = uint32_t(list.size()) - l0;
    if (!D) return;
    f.dmax = std::max(f.dmax, int(D));
    if (kind) f.dmax_same = std::max(f.dmax_same, int(D));
    jobs.push_back({l0, D, spect, count, c.w0, uint32_t(c.pairs.size()), kind, 0});
  };
  auto V = [&](int x0, int x1, int y0, int y1) {  // forward-ordered two-body value, x0 < x1, y0 < y1
    return x0 < y0 || (x0 == y0 && x1 <= y1) ? H.V(x0, x1, y0, y1) : H.V(y0, y1, x0, x1);
  };
  auto e1 = [&](int x, int y) { return H.e1[std::min(x, y) * ns + std::max(x, y)]; };

  // neutron + proton pairs by (2m, parity); the one-body terms of a neutron
  // move count once per proton of the determinant, so each pair takes 1 / kp of
  // them, and 1 / kn of a proton's
  std::map<std::pair<int, int>, Chan> pn;
  for (int x = 0; x < nn; ++x)
    for (int y = 0; y < np; ++y)
      pn[{m2[x] + m2[nn + y], par[x] ^ par[nn + y]}].pairs.push_back(uint16_t(x | (y << 8)));
  for (auto& kv : pn) {
    const auto& l = kv.second.pairs;
    if (l.size() > 256) return nullptr;
    kv.second.w0 = uint32_t(w.size());
    for (uint16_t p : l)
      for (uint16_t q : l) {
        const int x = p & 0xff, y = nn + (p >> 8), x2 = q & 0xff, y2 = nn + (q >> 8);
        double v = V(x, y, x2, y2);
        if (y == y2) v += e1(x, x2) / kp;
        if (x == x2) v += e1(y, y2) / kn;
        w.push_back(std::fabs(v) >= kFDrop ? v : 0.0);
      }
  }
  // The species with fewer cores gives the jobs' cores and the other one the
  // spectators, so that a job's matrix serves as many spectators as possible
  // (fp 5 + 2, cores 4845 and 20: 16 spectators a tile are full that way round
  // only).
  const Cores cores[2] = {make_cores(nn, kn - 1, m2, par), make_cores(np, kp - 1, m2 + nn, par + nn)};
  const int cs = cores[0].mask.size() <= cores[1].mask.size() ? 0 : 1, ss = 1 - cs;  // core and spectator species
  const int norb[2] = {nn, np}, npart[2] = {kn, kp};
  auto offset_of = [&](int sp, uint32_t m) {  // first row of a neutron configuration, rank of a proton one
    return sp ? uint32_t(b.h_pcrank[colex_host(m, b.h_binom)]) : start_of(m);
  };
  f.cols = norb[ss];
  std::vector<uint32_t> stab(cores[ss].mask.size() * f.cols, ~0u);
  for (size_t i = 0; i < cores[ss].mask.size(); ++i)
    for (int y = 0; y < f.cols; ++y) {
      const uint32_t m = cores[ss].mask[i];
      if ((m >> y) & 1) continue;
      const uint32_t r = offset_of(ss, m | (1u << y)), pos = uint32_t(popc(m & ((1u << y) - 1)));
      if (r != ~0u) stab[i * f.cols + y] = r | (pos << kFPosBit);
    }
  std::vector<uint32_t> first(norb[cs]);
  for (auto& gc : cores[cs].group)
    for (uint32_t i = 0; i < gc.second.second; ++i) {
      const uint32_t core = cores[cs].mask[gc.second.first + i];
      for (int x = 0; x < norb[cs]; ++x) first[x] = ((core >> x) & 1) ? ~0u : offset_of(cs, core | (1u << x));
      for (auto& gs : cores[ss].group) {
        const auto it =
            pn.find({b.twom - gc.first.first - gs.first.first, b.parity ^ gc.first.second ^ gs.first.second});
        if (it == pn.end()) continue;
        const auto& l = it->second.pairs;
        const uint32_t l0 = uint32_t(list.size());
        for (size_t k = 0; k < l.size(); ++k) {
          const uint32_t x = cs ? l[k] >> 8 : l[k] & 0xff, y = cs ? l[k] & 0xff : l[k] >> 8;
          if (first[x] == ~0u) continue;
          const uint32_t pos = uint32_t(popc(core & ((1u << x) - 1)));
          list.push_back({first[x], uint32_t(k) | (y << 8) | (pos * npart[ss] << 16) | (pos << 31)});
        }
        add_job(l0, gs.second.first, gs.second.second, it->second, 0);
      }
    }

  // pairs of one species: cores without two particles
  std::vector<uint32_t> spect;
  std::map<uint32_t, std::pair<uint32_t, uint32_t>> spect_of;  // proton class -> its blocks' starts
  for (int i = 0; i < nblocks; ++i) {
    auto& q = spect_of[b.h_bclass[i]];
    ++q.second;
  }
  {
    uint32_t at = 0;
    for (auto& kv : spect_of) {
      kv.second.first = at;
      at += kv.second.second;
    }
    spect.resize(at);
    std::map<uint32_t, uint32_t> fill;
    for (int i = 0; i < nblocks; ++i) {
      const uint32_t c = b.h_bclass[i];
      spect[spect_of[c].first + fill[c]++] = uint32_t(b.h_bstart[i]);
    }
  }
  std::map<std::pair<int, int>, uint32_t> class_of;  // (2m, parity) of the protons -> class
  for (size_t c = 0; c + 1 < b.h_cstart.size(); ++c) {
    if (b.h_cstart[c] == b.h_cstart[c + 1]) continue;
    int sm = 0, sp = 0;
    for (uint32_t t = b.h_cmasks[b.h_cstart[c]]; t; t &= t - 1) {
      sm += m2[nn + __builtin_ctz(t)];
      sp ^= par[nn + __builtin_ctz(t)];
    }
    class_of[{sm, sp}] = uint32_t(c);
  }
  for (int sp = 0; sp < 2; ++sp) {
    const int no = norb[sp], k = npart[sp], g0 = sp ? nn : 0;
    const int slot0 = kn * kp + (sp ? kn * (kn - 1) / 2 : 0);
    if (k < 2) continue;
    std::map<std::pair<int, int>, Chan> same;
    for (int x = 0; x < no; ++x)
      for (int y = x + 1; y < no; ++y)
        same[{m2[g0 + x] + m2[g0 + y], par[g0 + x] ^ par[g0 + y]}].pairs.push_back(uint16_t(x | (y << 8)));
    for (auto& kv : same) {
      const auto& l = kv.second.pairs;
      if (l.size() > 256) return nullptr;
      kv.second.w0 = uint32_t(w.size());
      for (uint16_t p : l)
        for (uint16_t q : l) {
          const double v = V(g0 + (p & 0xff), g0 + (p >> 8), g0 + (q & 0xff), g0 + (q >> 8));
          w.push_back(std::fabs(v) >= kFDrop ? v : 0.0);
        }
    }
    const Cores two = make_cores(no, k - 2, m2 + g0, par + g0);
    for (auto& gr : two.group)
      for (auto& chn : same) {
        const std::pair<int, int> full{gr.first.first + chn.first.first, gr.first.second ^ chn.first.second};
        const std::pair<int, int> protons =
            sp ? full : std::pair<int, int>{b.twom - full.first, b.parity ^ full.second};
        const auto cl = class_of.find(protons);
        if (cl == class_of.end()) continue;
        const uint32_t len = b.h_cstart[cl->second + 1] - b.h_cstart[cl->second];
        const auto so = spect_of.find(cl->second);
        if (sp && so == spect_of.end()) continue;
        const auto& l = chn.second.pairs;
        for (uint32_t i = 0; i < gr.second.second; ++i) {
          const uint32_t core = two.mask[gr.second.first + i];
          const uint32_t l0 = uint32_t(list.size());
          for (size_t q = 0; q < l.size(); ++q) {
            const int x = l[q] & 0xff, y = l[q] >> 8;
            if (((core >> x) | (core >> y)) & 1) continue;
            const uint32_t m = core | (1u << x) | (1u << y);
            const int px = popc(core & ((1u << x) - 1)), py = popc(core & ((1u << y) - 1));
            // positions of the two in the full configuration, px <= py: slot of the pair (px, py + 1)
            const int i0 = px, i1 = py + 1;
            const int slot = slot0 + i0 * k - i0 * (i0 + 1) / 2 + (i1 - i0 - 1);
            const uint32_t r = offset_of(sp, m);
            if (r == ~0u) continue;
            list.push_back({r, uint32_t(q) | (uint32_t(slot) << 16) | (uint32_t(px + py) << 31)});
          }
          add_job(l0, sp ? so->second.first : ~0u, sp ? so->second.second : len, chn.second, 1);
        }
      }
  }
  if (f.dmax > kFMaxPairs || f.dmax_same > kFPairs || w.size() >= (1ull << 31) || list.size() >= (1ull << 32))
    return nullptr;
  // at least 16 spectators a chunk beside the largest matrix
  f.smem32 = std::max(kFSmem, int(sizeof(FHead32)) + f.dmax * fact_tiles(f.dmax) * 64 +
                                  16 * (f.dmax * 36 + 2 * f.cols * 4));
  if (f.smem32 > kSmemMax) return nullptr;
  // few jobs: split their spectators (whole tiles of 16, or 64 rows) until there are some per CTA slot
  constexpr size_t kEnough = 152 * 16;
  for (uint32_t kind = 0; kind < 2; ++kind) {
    size_t have = 0;
    for (const FJob& j : jobs) have += j.kind == kind;
    if (!have || 2 * have > kEnough) continue;
    const uint32_t parts = uint32_t(kEnough / have), unit = kind ? 64 : 16;
    std::vector<FJob> cut;
    for (const FJob& j : jobs) {
      const uint32_t units = (j.count + unit - 1) / unit, np1 = j.kind == kind ? std::min(parts, units) : 1;
      for (uint32_t p = 0; p < np1; ++p) {
        FJob q = j;
        const uint32_t at = np1 == 1 ? 0 : uint32_t(uint64_t(units) * p / np1) * unit;
        const uint32_t end = p + 1 == np1 ? j.count : uint32_t(uint64_t(units) * (p + 1) / np1) * unit;
        q.count = end - at;
        if (q.spect == ~0u) q.first += at;
        else q.spect += at;
        cut.push_back(q);
      }
    }
    jobs.swap(cut);
  }
  // neutron + proton jobs first, each kind largest first
  auto macs = [](const FJob& j) { return double(j.npair) * ((j.npair + 7) / 8 * 8) * ((j.count + 15) / 16 * 16); };
  std::stable_sort(jobs.begin(), jobs.end(), [&](const FJob& p, const FJob& q) {
    return p.kind != q.kind ? p.kind < q.kind : macs(p) > macs(q);
  });
  for (const FJob& j : jobs) {
    (j.kind ? f.macs_same : f.macs) += macs(j);
    f.njobs_pn += j.kind == 0;
  }
  f.njobs = jobs.size();
  // Time of one product in us, fitted to sd and fp systems of 28 to 1,963,461
  // rows (fp 4 + 4: 0.84 + 0.26 + 0.26 ms; sd 6 + 6: 98 + 46 + 27 us): the
  // multiply-adds and the start of each job, and the partial sums read back.
  f.est_us = 12 + 4.7e-7 * f.macs + 6.5e-3 * f.njobs_pn + 3e-7 * f.macs_same + 7e-3 * (f.njobs - f.njobs_pn) +
             double(slots) * b.n * 32 / 6.5e6;
  if (f.est_us > other_us) return nullptr;
  f.jobs.upload(jobs, s);
  f.list.upload(list, s);
  f.stab.upload(stab, s);
  f.spect.upload(spect, s);
  const std::vector<float> wf(w.begin(), w.end());
  f.wf.upload(wf, s);
  CG_CUDA(cudaStreamSynchronize(s));
  return fp;
}

}  // namespace

std::shared_ptr<FactoredOp> factored_build(const System& sys, const Operator& op, const Basis& b, double other_us,
                                           cudaStream_t s) {
  try {
    return build_tables(sys, op, b, other_us, s);
  } catch (const Error& e) {
    if (e.code != CG_ERR_NOMEM) throw;
    return nullptr;
  }
}

bool factored_ready(const Hamiltonian& h) {
  const FactoredOp& f = *h.fact;
  if (f.z.p || !f.n) return true;
  try {
    f.z.alloc(uint64_t(f.slots) * f.n * 32);
  } catch (const Error& e) {
    if (e.code != CG_ERR_NOMEM) throw;
    h.fact_failed = true;
  }
  return f.z.p;
}

void factored_product_f32(const FactoredOp& f, const float* x, float* y, int ldy, int m, cudaStream_t s) {
  if (m < 1 || m > 8) throw Error(CG_ERR_ARG, "factored product: too many vectors for one pass");
  if (ldy < m) throw Error(CG_ERR_ARG, "leading dimension smaller than the vector count");
  if (reinterpret_cast<uintptr_t>(x) % 32) throw Error(CG_ERR_ARG, "factored product needs 32-byte aligned rows");
  if (!f.n) return;
  FArgs a{f.n, f.cols, f.jobs.p, f.list.p, f.stab.p, f.spect.p};
  const unsigned char* xb = reinterpret_cast<const unsigned char*>(x);
  CG_CUDA(cudaFuncSetAttribute(k_fact32, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
  k_fact32<<<unsigned(f.njobs_pn), kFW * 32, f.smem32, s>>>(a, f.wf.p, xb, f.z.p, f.smem32);
  CG_CUDA(cudaGetLastError());
  count_launch();
  if (f.njobs > f.njobs_pn) {
    a.jobs += f.njobs_pn;
    k_pair32<<<unsigned(f.njobs - f.njobs_pn), 128, 0, s>>>(a, f.wf.p, xb, f.z.p);
    CG_CUDA(cudaGetLastError());
    count_launch();
  }
  const bool vec = m == 8 && reinterpret_cast<uintptr_t>(y) % 16 == 0 && ldy % 4 == 0;
  k_fsum<<<unsigned((2 * f.n + 255) / 256), 256, 0, s>>>(f.n, f.slots, reinterpret_cast<const float4*>(f.z.p), y, ldy,
                                                         m, vec);
  CG_CUDA(cudaGetLastError());
  count_launch();
}

}  // namespace cg
