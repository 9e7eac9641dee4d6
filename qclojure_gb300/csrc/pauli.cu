// <psi|P|psi> for many Pauli strings of one state (hamiltonian.clj:82-114).
//
// (P psi)_i = (-i)^ny (-1)^popc(i & z) psi_{i ^ x}, so strings with the same x mask (and the
// same parity of their Y count) are signed sums of the same values: with x = 0, of the
// probabilities |a_i|^2 over all i; otherwise, over the pairs (i, i ^ x) with the top x bit of i
// clear, of Re or Im of conj(a_i) a_{i^x} (each pair counts twice). Pair index q is i without
// that bit; a string's sign is the parity of q & zq.
//
// What bounds it: the FP64 pipe (two lanes per clock and SM on this part). One kernel per
// string cost three to four FP64 instructions for the value and seven for a TwoSum per
// amplitude, and one host round trip per string: 24 qubits, complex128, a Heisenberg chain of
// 93 strings took 93 x 320 us. Here a group's values are formed once for all of its strings (two
// FP64 instructions each), summed exactly in fixed point on the integer pipes (fixed_sum.cuh), and
// all groups run in one launch; every string's sum is that of its rounded values, in any company:
//   * up to two strings per group (XX and YY on a pair): each thread adds its 16 values of a tile
//     to both sums with their signs, then one TwoSum takes each;
//   * more strings (the Z and ZZ terms): a Walsh-Hadamard transform of the tile over 8 of its 12
//     index bits (4 in registers, 4 after an exchange through shared memory), of the upper and the
//     lower integers in turn, then one thread per string adds its 16 remaining signed values and
//     does one TwoSum per tile of 4096.
// 24 qubits, complex128, the 93 strings: 2.60 ms (3.28 ms with the 16 values added in FP64 before
// a TwoSum, which also lost what the TwoSum is for: cancelling terms were off by ulps of the terms).
// Neighbouring CTAs work on the same chunk of different groups, so the state is read from L2 by
// all but the first of them.
#include <algorithm>
#include <cstring>
#include <map>
#include <string>
#include <utility>
#include <vector>

#include "fixed_sum.cuh"
#include "qgpu_internal.h"

namespace qg {

namespace {

constexpr int kTileBits = 12;      // values per tile: 16 per thread, 256 threads
constexpr int kGroupStrings = 256; // strings per group at most (one thread each)
constexpr int kPitch = 256 + 16;   // words per transform row: t + t / 16, free of bank conflicts

struct PauliGroup {
  uint64_t xm;
  int32_t hb;      // top bit of xm (-1: x = 0)
  int32_t imag;    // Im instead of Re (odd number of Y)
  int32_t t0, nt;  // its strings
};
struct PauliString {
  uint64_t zq;
  double factor;   // applied to the sum: 1 for x = 0, 2 or -2 for pairs
};

__device__ __forceinline__ void two_sum(double& s, double& c, double x) {
  const double t = __dadd_rn(s, x);
  const double bp = __dsub_rn(t, s);
  c = __dadd_rn(c, __dadd_rn(__dsub_rn(s, __dsub_rn(t, bp)), __dsub_rn(x, bp)));
  s = t;
}

// (double)f with integer instructions (the conversion runs at the FP64 rate)
__device__ __forceinline__ double widen(float f) {
  const uint32_t b = __float_as_uint(f), e = (b >> 23) & 0xFFu;
  if (e == 0xFFu || (e == 0u && (b & 0x7FFFFFu))) return (double)f;
  const uint32_t hi = (b & 0x80000000u) | (e ? ((b & 0x7FFFFFFFu) >> 3) + (896u << 20) : 0u);
  return __hiloint2double((int)hi, (int)(b << 29));
}
__device__ __forceinline__ double2 amp(const double2* s, uint64_t i) { return __ldg(s + i); }
__device__ __forceinline__ double2 amp(const float2* s, uint64_t i) {
  const float2 v = __ldg(s + i);
  return make_double2(widen(v.x), widen(v.y));
}
__device__ __forceinline__ double prob(const double2* s, uint64_t i) {
  const double2 v = __ldg(s + i);
  return fma(v.x, v.x, __dmul_rn(v.y, v.y));
}
__device__ __forceinline__ double prob(const float2* s, uint64_t i) {
  const float2 v = __ldg(s + i);
  return __dadd_rn(qg_sq_float(v.x), qg_sq_float(v.y));
}

template <typename T>
__device__ __forceinline__ void tile_values(const T* __restrict__ s, const PauliGroup& g, uint64_t q0, uint64_t count,
                                            double (&v)[16]) {
  if (g.hb < 0) {
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const uint64_t q = q0 + (uint64_t)r * 256;
      v[r] = q < count ? prob(s, q) : 0.0;
    }
    return;
  }
  const uint64_t low = (1ULL << g.hb) - 1;
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    const uint64_t q = q0 + (uint64_t)r * 256;
    if (q < count) {
      const uint64_t i = ((q & ~low) << 1) | (q & low);
      const double2 a = amp(s, i), b = amp(s, i ^ g.xm);
      v[r] = g.imag ? fma(a.x, b.y, -__dmul_rn(a.y, b.x)) : fma(a.x, b.x, __dmul_rn(a.y, b.y));
    } else {
      v[r] = 0.0;
    }
  }
}

// the parity of r & z for r = 0..15, as a bit pattern
__device__ __forceinline__ uint32_t parities(uint32_t z) {
  return ((z & 1) ? 0xAAAAu : 0u) ^ ((z & 2) ? 0xCCCCu : 0u) ^ ((z & 4) ? 0xF0F0u : 0u) ^ ((z & 8) ? 0xFF00u : 0u);
}

__device__ __forceinline__ uint32_t top_key(const double (&v)[16]) {
  uint32_t key = 0;
#pragma unroll
  for (int r = 0; r < 16; ++r) key = max(key, qg_fix_key(v[r]));
  return key;
}

// sums and differences over 4 index bits
__device__ __forceinline__ void transform(int64_t (&v)[16]) {
#pragma unroll
  for (int o = 1; o < 16; o <<= 1)
#pragma unroll
    for (int r = 0; r < 16; ++r)
      if (!(r & o)) {
        const int64_t x = v[r], y = v[r + o];
        v[r] = x + y;
        v[r + o] = x - y;
      }
}

template <typename T>
__global__ void __launch_bounds__(256, 3) k_pauli_sums(const T* __restrict__ s, int n,
                                                       const PauliGroup* __restrict__ groups,
                                                       const PauliString* __restrict__ strings, int ngroups,
                                                       int nchunks, double2* __restrict__ partial) {
  __shared__ int64_t sh[16 * kPitch];
  __shared__ uint32_t keys[8];
  const int chunk = (int)(blockIdx.x / (unsigned)ngroups);
  const PauliGroup g = groups[blockIdx.x - (unsigned)chunk * (unsigned)ngroups];
  const uint64_t count = (1ULL << n) >> (g.hb < 0 ? 0 : 1);
  const uint64_t tiles = (count + (1ULL << kTileBits) - 1) >> kTileBits;
  const uint64_t w0 = tiles * (uint64_t)chunk / (uint64_t)nchunks, w1 = tiles * (uint64_t)(chunk + 1) / (uint64_t)nchunks;
  const int tid = (int)threadIdx.x;
  if (g.nt <= 2) {
    const uint64_t z0 = strings[g.t0].zq, z1 = strings[g.t0 + g.nt - 1].zq;
    const uint32_t p0 = parities((uint32_t)(z0 >> 8)), p1 = parities((uint32_t)(z1 >> 8));  // register positions: bits 8..11
    double s0 = 0, c0 = 0, s1 = 0, c1 = 0;
    for (uint64_t t = w0; t < w1; ++t) {
      const uint64_t q0 = (t << kTileBits) + (uint64_t)tid;
      double v[16];
      tile_values(s, g, q0, count, v);
      const int E = qg_fix_exponent(top_key(v));
      const uint32_t t0 = (uint32_t)__popcll(q0 & z0) & 1u, t1 = (uint32_t)__popcll(q0 & z1) & 1u;
      int64_t h0 = 0, l0 = 0, h1 = 0, l1 = 0;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const qg_fixed x = qg_fix(v[r], E, ((p0 >> r) & 1u) ^ t0);
        const int64_t other = -(int64_t)((((p0 ^ p1) >> r) & 1u) ^ t0 ^ t1);  // string 1's sign against string 0's
        h0 += x.h;
        l0 += x.l;
        h1 += (x.h ^ other) - other;
        l1 += (x.l ^ other) - other;
      }
      two_sum(s0, c0, qg_fix_hi(h0, E));
      c0 = __dadd_rn(c0, qg_fix_lo(l0, E));
      if (g.nt == 2) {
        two_sum(s1, c1, qg_fix_hi(h1, E));
        c1 = __dadd_rn(c1, qg_fix_lo(l1, E));
      }
    }
    __shared__ double2 red[2][8];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      double ss = k ? s1 : s0, cc = k ? c1 : c0;
      if (k >= g.nt) break;
      for (int o = 16; o > 0; o >>= 1) {
        const double us = __shfl_down_sync(0xffffffffu, ss, o), uc = __shfl_down_sync(0xffffffffu, cc, o);
        two_sum(ss, cc, us);
        cc = __dadd_rn(cc, uc);
      }
      if ((tid & 31) == 0) red[k][tid >> 5] = make_double2(ss, cc);
    }
    __syncthreads();
    if (tid < g.nt) {
      double ss = red[tid][0].x, cc = red[tid][0].y;
      for (int w = 1; w < 8; ++w) {
        two_sum(ss, cc, red[tid][w].x);
        cc = __dadd_rn(cc, red[tid][w].y);
      }
      partial[(size_t)(g.t0 + tid) * nchunks + chunk] = make_double2(ss, cc);
    }
    return;
  }
  const bool mine = tid < g.nt;
  const uint64_t zq = mine ? strings[g.t0 + tid].zq : 0;
  const int row = (int)(zq >> 8) & 15, col = (int)zq & 15;
  const uint32_t ph = parities((uint32_t)(zq >> 4));
  double acc = 0, comp = 0;
  for (uint64_t t = w0; t < w1; ++t) {
    const uint32_t ts = (uint32_t)__popcll((t << kTileBits) & zq) & 1u;
    int E = 0;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {  // the upper integers, then the lower ones of the same values
      double v[16];
      tile_values(s, g, (t << kTileBits) + (uint64_t)tid, count, v);
      if (part == 0) {
        const uint32_t key = __reduce_max_sync(0xffffffffu, top_key(v));
        if ((tid & 31) == 0) keys[tid >> 5] = key;
        __syncthreads();  // and the previous tile's readers are done
        uint32_t top = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) top = max(top, keys[w]);
        E = qg_fix_exponent(top);
      }
      int64_t x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const qg_fixed f = qg_fix(v[r], E, 0);
        x[r] = part ? f.l : f.h;
      }
      transform(x);
      if (part) __syncthreads();  // the readers of the upper integers are done
#pragma unroll
      for (int r = 0; r < 16; ++r) sh[r * kPitch + tid + (tid >> 4)] = x[r];
      __syncthreads();
      int64_t* mr = sh + (tid >> 4) * kPitch + (tid & 15) * 17;  // 16 values of one row, index bits 0..3
#pragma unroll
      for (int l = 0; l < 16; ++l) x[l] = mr[l];
      transform(x);
#pragma unroll
      for (int l = 0; l < 16; ++l) mr[l] = x[l];
      __syncthreads();
      if (mine) {
        int64_t sum = 0;
#pragma unroll
        for (int h = 0; h < 16; ++h) {
          const int64_t f = -(int64_t)(((ph >> h) & 1u) ^ ts);
          sum += (sh[row * kPitch + h * 17 + col] ^ f) - f;
        }
        if (part) comp = __dadd_rn(comp, qg_fix_lo(sum, E));
        else two_sum(acc, comp, qg_fix_hi(sum, E));
      }
    }
  }
  if (mine) partial[(size_t)(g.t0 + tid) * nchunks + chunk] = make_double2(acc, comp);
}

// one warp per string: its chunks' (sum, compensation) pairs in a fixed order
__global__ void __launch_bounds__(128) k_pauli_fold(const double2* __restrict__ partial,
                                                    const PauliString* __restrict__ strings, int nstrings, int nchunks,
                                                    double* __restrict__ out) {
  const int k = (int)(blockIdx.x * 4 + (threadIdx.x >> 5)), lane = (int)threadIdx.x & 31;
  if (k >= nstrings) return;
  double s = 0, c = 0;
  for (int i = lane; i < nchunks; i += 32) {
    const double2 p = partial[(size_t)k * nchunks + i];
    two_sum(s, c, p.x);
    c = __dadd_rn(c, p.y);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double us = __shfl_down_sync(0xffffffffu, s, o), uc = __shfl_down_sync(0xffffffffu, c, o);
    two_sum(s, c, us);
    c = __dadd_rn(c, uc);
  }
  if (lane == 0) out[k] = strings[k].factor * __dadd_rn(s, c);
}

}  // namespace

bool PauliPlan::build(int n, int count, const char* text) {
  struct Key {
    uint64_t x;
    int imag;
    bool operator<(const Key& o) const { return x != o.x ? x < o.x : imag < o.imag; }
  };
  std::map<Key, std::vector<std::pair<int, PauliString>>> by;
  for (int k = 0; k < count; ++k) {
    uint64_t x = 0, z = 0;
    int ny = 0;
    for (int q = 0; q < n; ++q) {
      const uint64_t b = 1ULL << (n - 1 - q);
      const char ch = text[(size_t)k * n + q];
      if (ch == 'X') x |= b;
      else if (ch == 'Y') { x |= b; z |= b; ++ny; }
      else if (ch == 'Z') z |= b;
      else if (ch != 'I') return false;
    }
    PauliString p{z, 1.0};
    if (x) {
      const int hb = 63 - __builtin_clzll(x);
      p.zq = (z & ((1ULL << hb) - 1)) | ((z >> (hb + 1)) << hb);
      p.factor = (ny & 2) ? -2.0 : 2.0;
    }
    by[Key{x, x ? (ny & 1) : 0}].push_back({k, p});
  }
  std::vector<PauliGroup> groups;
  std::vector<PauliString> strings;
  order.assign((size_t)count, 0);
  for (auto& [key, v] : by) {
    for (size_t i = 0; i < v.size(); i += kGroupStrings) {
      const int nt = (int)std::min<size_t>(kGroupStrings, v.size() - i);
      groups.push_back(PauliGroup{key.x, key.x ? 63 - __builtin_clzll(key.x) : -1, key.imag, (int32_t)strings.size(), nt});
      for (int j = 0; j < nt; ++j) {
        order[(size_t)v[i + j].first] = (int)strings.size();
        strings.push_back(v[i + j].second);
      }
    }
  }
  ngroups = (int)groups.size();
  nstrings = count;
  // about four waves of three CTAs per SM over all groups; at least four tiles per CTA (each ends
  // with a reduction) where that still fills the device
  const uint64_t tiles = n > kTileBits ? (1ULL << (n - kTileBits)) : 1;
  const uint64_t wave = 152 * 3, ng = (uint64_t)std::max(1, ngroups);
  uint64_t ch = std::min(tiles, std::max<uint64_t>(1, wave * 4 / ng));
  if (tiles / ch < 4 && tiles / 4 * ng >= wave) ch = tiles / 4;
  nchunks = (int)ch;
  string_bytes = sizeof(PauliString) * strings.size();
  table.resize(string_bytes + sizeof(PauliGroup) * groups.size());
  std::memcpy(table.data(), strings.data(), string_bytes);
  std::memcpy(table.data() + string_bytes, groups.data(), sizeof(PauliGroup) * groups.size());
  partial_bytes = sizeof(double2) * (size_t)count * (size_t)nchunks;
  return true;
}

cudaError_t launch_pauli_plan(const void* s, int precision, int n, const PauliPlan& p, const void* d_table,
                              void* d_partial, double* d_out, cudaStream_t st) {
  const PauliString* ds = reinterpret_cast<const PauliString*>(d_table);
  const PauliGroup* dg = reinterpret_cast<const PauliGroup*>(static_cast<const unsigned char*>(d_table) + p.string_bytes);
  const unsigned grid = (unsigned)p.ngroups * (unsigned)p.nchunks;
  if (precision == QG_C64)
    k_pauli_sums<float2><<<grid, 256, 0, st>>>((const float2*)s, n, dg, ds, p.ngroups, p.nchunks, (double2*)d_partial);
  else
    k_pauli_sums<double2><<<grid, 256, 0, st>>>((const double2*)s, n, dg, ds, p.ngroups, p.nchunks, (double2*)d_partial);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_pauli_fold<<<(unsigned)(p.nstrings + 3) / 4, 128, 0, st>>>((const double2*)d_partial, ds, p.nstrings, p.nchunks, d_out);
  count_launch(2);
  return cudaGetLastError();
}

}  // namespace qg
