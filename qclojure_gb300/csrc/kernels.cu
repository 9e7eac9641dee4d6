// sm_103a kernels of libqgpu.so.
//
// State layout in HBM: 2^n interleaved complex amplitudes (double2 for c128,
// float2 for c64), basis index i, qubit q <-> bit (n-1-q) of i.
//
// Arithmetic: every 2x2 class, phase and collapse multiplies with the same
// rounded products and sums the reference's complex multiply and dense row sum
// form (src/org/soulspace/qclojure/domain/gate.clj:384-395,
// src/org/soulspace/qclojure/domain/math/fastmath/complex_linear_algebra.clj:408-431),
// written with explicit __dmul_rn/__dadd_rn so nothing is contracted into an FMA.
// The complex128 path therefore reproduces the CPU restatement bit for bit, and
// the plain (one pass per gate) and tiled (many gates per pass) executors give
// identical amplitudes. Dense fused blocks use FMA and are checked to tolerance.
#include <algorithm>
#include <atomic>
#include <cstdio>

#include "fixed_sum.cuh"
#include "qgpu_internal.h"

namespace qg {

namespace {

constexpr int kSMs = 152;

std::atomic<unsigned long long> g_launches{0};
inline void counted(int k = 1) { g_launches.fetch_add((unsigned long long)k, std::memory_order_relaxed); }

template <typename R> struct C2;
template <> struct C2<double> { using T = double2; };
template <> struct C2<float> { using T = float2; };

__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_(float a, float b) { return __fsub_rn(a, b); }

// reference complex multiply g*x: (g.re x.re - g.im x.im, g.re x.im + g.im x.re)
template <typename V, typename R>
__device__ __forceinline__ V cmul(R gr, R gi, V x) {
  V r;
  r.x = sub_(mul_(gr, x.x), mul_(gi, x.y));
  r.y = add_(mul_(gr, x.y), mul_(gi, x.x));
  return r;
}
template <typename V>
__device__ __forceinline__ V cadd(V a, V b) {
  V r;
  r.x = add_(a.x, b.x);
  r.y = add_(a.y, b.y);
  return r;
}

template <typename R>
struct Mat {
  R m[8];
};

template <typename R>
Mat<R> to_mat(const double* m) {
  Mat<R> r;
  for (int k = 0; k < 8; ++k) r.m[k] = (R)m[k];
  return r;
}

// 2x2 application per class; y0,y1 from x0,x1.
template <int CLS, typename V, typename R>
__device__ __forceinline__ void u2_apply(const R* m, V x0, V x1, V& y0, V& y1) {
  if (CLS == U2_GENERAL) {
    y0 = cadd(cmul(m[0], m[1], x0), cmul(m[2], m[3], x1));
    y1 = cadd(cmul(m[4], m[5], x0), cmul(m[6], m[7], x1));
  } else if (CLS == U2_REAL) {
    y0.x = add_(mul_(m[0], x0.x), mul_(m[2], x1.x));
    y0.y = add_(mul_(m[0], x0.y), mul_(m[2], x1.y));
    y1.x = add_(mul_(m[4], x0.x), mul_(m[6], x1.x));
    y1.y = add_(mul_(m[4], x0.y), mul_(m[6], x1.y));
  } else if (CLS == U2_RXLIKE) {
    // m0=(a,0) m1=(0,b) m2=(0,c) m3=(d,0)
    y0.x = sub_(mul_(m[0], x0.x), mul_(m[3], x1.y));
    y0.y = add_(mul_(m[0], x0.y), mul_(m[3], x1.x));
    y1.x = sub_(mul_(m[6], x1.x), mul_(m[5], x0.y));
    y1.y = add_(mul_(m[5], x0.x), mul_(m[6], x1.y));
  } else if (CLS == U2_DIAG) {
    y0 = cmul(m[0], m[1], x0);
    y1 = cmul(m[6], m[7], x1);
  } else if (CLS == U2_ANTIDIAG) {
    y0 = cmul(m[2], m[3], x1);
    y1 = cmul(m[4], m[5], x0);
  } else if (CLS == U2_X) {
    y0 = x1;
    y1 = x0;
  } else {  // U2_IMAG_ANTI: m1=(0,s1), m2=(0,s2), s=+-1: (0,s)*x = (-s x.im, s x.re)
    if (m[3] > 0) { y0.x = -x1.y; y0.y = x1.x; } else { y0.x = x1.y; y0.y = -x1.x; }
    if (m[5] > 0) { y1.x = -x0.y; y1.y = x0.x; } else { y1.x = x0.y; y1.y = -x0.x; }
  }
}

template <int CLS, typename V, typename R>
__device__ __forceinline__ V phase_apply(const R* m, V x) {
  if (CLS == PH_GENERAL) return cmul(m[0], m[1], x);
  V r;
  if (CLS == PH_NEG) { r.x = -x.x; r.y = -x.y; }
  else if (CLS == PH_I) { r.x = -x.y; r.y = x.x; }
  else { r.x = x.y; r.y = -x.x; }
  return r;
}

// Insert bits: positions ascending; bits in setmask become 1, the others 0.
struct Fixed {
  int n;
  int pos[8];
  uint64_t setmask;
};
__device__ __forceinline__ uint64_t expand(uint64_t j, const Fixed& f) {
#pragma unroll 1
  for (int i = 0; i < f.n; ++i) {
    int b = f.pos[i];
    uint64_t lo = j & ((1ULL << b) - 1);
    j = ((j >> b) << (b + 1)) | lo;
  }
  return j | f.setmask;
}

Fixed make_fixed(uint64_t zero_bits, uint64_t one_bits) {
  Fixed f;
  f.n = 0;
  f.setmask = one_bits;
  uint64_t all = zero_bits | one_bits;
  for (int b = 0; b < 64 && f.n < 8; ++b)
    if (all & (1ULL << b)) f.pos[f.n++] = b;
  return f;
}

inline int grid_for(uint64_t work, int threads) {
  uint64_t g = (work + threads - 1) / threads;
  uint64_t cap = (uint64_t)kSMs * 8;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

// ---------------------------------------------------------------------------
// Plain kernels: one gate, one HBM pass, grid-stride.
// ---------------------------------------------------------------------------
template <int CLS, typename R>
__global__ void __launch_bounds__(256) k_u2(typename C2<R>::T* __restrict__ s, uint64_t work, int t, Fixed f,
                                            Mat<R> m) {
  using V = typename C2<R>::T;
  const uint64_t tb = 1ULL << t;
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < work; j += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t i0 = expand(j, f);
    V x0 = s[i0], x1 = s[i0 | tb], y0, y1;
    u2_apply<CLS, V, R>(m.m, x0, x1, y0, y1);
    s[i0] = y0;
    s[i0 | tb] = y1;
  }
}

template <int CLS, typename R>
__global__ void __launch_bounds__(256) k_phase(typename C2<R>::T* __restrict__ s, uint64_t work, Fixed f, Mat<R> m) {
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < work; j += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t i = expand(j, f);
    s[i] = phase_apply<CLS>(m.m, s[i]);
  }
}

template <typename R>
__global__ void __launch_bounds__(256) k_swap(typename C2<R>::T* __restrict__ s, uint64_t work, uint64_t flip, Fixed f,
                                              int iswap) {
  using V = typename C2<R>::T;
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < work; j += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t i = expand(j, f), p = i ^ flip;
    V a = s[i], b = s[p];
    if (iswap) {
      V ra, rb;
      ra.x = -b.y; ra.y = b.x;   // i * b
      rb.x = -a.y; rb.y = a.x;   // i * a
      a = ra;
      b = rb;
      s[i] = a;
      s[p] = b;
    } else {
      s[i] = b;
      s[p] = a;
    }
  }
}

// kind: 0 blockade (popcount==1 -> ph), 1 parity (ph0/ph1)
template <int KIND, typename R>
__global__ void __launch_bounds__(256) k_diag_all(typename C2<R>::T* __restrict__ s, uint64_t N, uint64_t mask,
                                                  Mat<R> m) {
  using V = typename C2<R>::T;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    V x = s[i];
    if (KIND == 0) {
      if (__popcll(i & mask) == 1) s[i] = cmul(m.m[0], m.m[1], x);
    } else {
      if (__popcll(i & mask) & 1) s[i] = cmul(m.m[2], m.m[3], x);
      else s[i] = cmul(m.m[0], m.m[1], x);
    }
  }
}

template <typename R>
cudaError_t plain_op_t(void* sv, int n, const GOp& op, cudaStream_t st) {
  using V = typename C2<R>::T;
  V* s = (V*)sv;
  const int T = 256;
  const uint64_t N = 1ULL << n;
  switch (op.kind) {
    case OK_U2: {
      Fixed f = make_fixed(1ULL << op.t, op.cmask);
      uint64_t work = N >> f.n;
      Mat<R> m = to_mat<R>(op.m);
      int g = grid_for(work, T);
      switch (op.cls) {
        case U2_GENERAL: k_u2<U2_GENERAL, R><<<g, T, 0, st>>>(s, work, op.t, f, m); break;
        case U2_REAL: k_u2<U2_REAL, R><<<g, T, 0, st>>>(s, work, op.t, f, m); break;
        case U2_RXLIKE: k_u2<U2_RXLIKE, R><<<g, T, 0, st>>>(s, work, op.t, f, m); break;
        case U2_DIAG: k_u2<U2_DIAG, R><<<g, T, 0, st>>>(s, work, op.t, f, m); break;
        case U2_ANTIDIAG: k_u2<U2_ANTIDIAG, R><<<g, T, 0, st>>>(s, work, op.t, f, m); break;
        case U2_X: k_u2<U2_X, R><<<g, T, 0, st>>>(s, work, op.t, f, m); break;
        default: k_u2<U2_IMAG_ANTI, R><<<g, T, 0, st>>>(s, work, op.t, f, m); break;
      }
    } break;
    case OK_PHASE: {
      Fixed f = make_fixed(0, op.mask);
      uint64_t work = N >> f.n;
      Mat<R> m = to_mat<R>(op.m);
      int g = grid_for(work, T);
      switch (op.cls) {
        case PH_GENERAL: k_phase<PH_GENERAL, R><<<g, T, 0, st>>>(s, work, f, m); break;
        case PH_NEG: k_phase<PH_NEG, R><<<g, T, 0, st>>>(s, work, f, m); break;
        case PH_I: k_phase<PH_I, R><<<g, T, 0, st>>>(s, work, f, m); break;
        default: k_phase<PH_MINUS_I, R><<<g, T, 0, st>>>(s, work, f, m); break;
      }
    } break;
    case OK_SWAP: {
      Fixed f = make_fixed(1ULL << op.t2, (1ULL << op.t) | op.cmask);
      uint64_t work = N >> f.n;
      k_swap<R><<<grid_for(work, T), T, 0, st>>>(s, work, (1ULL << op.t) | (1ULL << op.t2), f, op.flags & 1);
    } break;
    case OK_BLOCKADE:
      k_diag_all<0, R><<<grid_for(N, T), T, 0, st>>>(s, N, op.mask, to_mat<R>(op.m));
      break;
    case OK_PARITY:
      k_diag_all<1, R><<<grid_for(N, T), T, 0, st>>>(s, N, op.mask, to_mat<R>(op.m));
      break;
    default:
      return cudaErrorInvalidValue;
  }
  counted();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Reductions. Per-thread TwoSum accumulation, warp/block combination of
// (sum, compensation) pairs, one pair per block written to d_part.
// ---------------------------------------------------------------------------
struct DD {
  double s, c;
};
__device__ __forceinline__ void two_sum_acc(DD& a, double x) {
  double t = __dadd_rn(a.s, x);
  double bp = __dsub_rn(t, a.s);
  double e = __dadd_rn(__dsub_rn(a.s, __dsub_rn(t, bp)), __dsub_rn(x, bp));
  a.s = t;
  a.c = __dadd_rn(a.c, e);
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  DD r = a;
  two_sum_acc(r, b.s);
  r.c = __dadd_rn(r.c, b.c);
  return r;
}
template <int NT>
__device__ __forceinline__ void block_reduce_store(DD v, double* d_part, int slot) {
  __shared__ DD red[NT / 32];
  for (int o = 16; o > 0; o >>= 1) {
    DD w;
    w.s = __shfl_down_sync(0xffffffffu, v.s, o);
    w.c = __shfl_down_sync(0xffffffffu, v.c, o);
    v = dd_add(v, w);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    DD a = red[0];
    for (int w = 1; w < NT / 32; ++w) a = dd_add(a, red[w]);
    d_part[2 * slot] = a.s;
    d_part[2 * slot + 1] = a.c;
  }
}

template <typename R>
__device__ __forceinline__ double p_of(typename C2<R>::T a) {
  if constexpr (sizeof(R) == 4) {
    // the squares of floats are exact doubles, built on the integer pipes (quant.cuh):
    // only the rounded sum is an FP64 instruction
    return __dadd_rn(qg_sq_float(a.x), qg_sq_float(a.y));
  } else {
    const double re = a.x, im = a.y;
    return __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
  }
}

// floor(p 2^62) on the integer pipes (quant.cuh): the FP64 product and conversion's value
__device__ __forceinline__ unsigned long long quant(double p) { return qg_quant62(p); }

template <typename R>
__global__ void __launch_bounds__(256) k_probs(const typename C2<R>::T* __restrict__ s, uint64_t N,
                                               double* __restrict__ p) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = p_of<R>(s[i]);
}

template <typename R>
__global__ void __launch_bounds__(256) k_norm2(const typename C2<R>::T* __restrict__ s, uint64_t N, double* d_part) {
  DD a{0, 0};
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x)
    two_sum_acc(a, p_of<R>(s[i]));
  block_reduce_store<256>(a, d_part, blockIdx.x);
}

template <typename R>
__global__ void __launch_bounds__(256) k_expect1q(const typename C2<R>::T* __restrict__ s, uint64_t N, int bit,
                                                  Mat<double> o, double* d_part) {
  DD acc{0, 0};
  const uint64_t half = N >> 1, tb = 1ULL << bit;
  for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < half; q += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t i0 = ((q >> bit) << (bit + 1)) | (q & (tb - 1));
    auto a = s[i0];
    auto b = s[i0 | tb];
    double x0r = a.x, x0i = a.y, x1r = b.x, x1i = b.y;
    double y0r = o.m[0] * x0r - o.m[1] * x0i + o.m[2] * x1r - o.m[3] * x1i;
    double y0i = o.m[0] * x0i + o.m[1] * x0r + o.m[2] * x1i + o.m[3] * x1r;
    double y1r = o.m[4] * x0r - o.m[5] * x0i + o.m[6] * x1r - o.m[7] * x1i;
    double y1i = o.m[4] * x0i + o.m[5] * x0r + o.m[6] * x1i + o.m[7] * x1r;
    two_sum_acc(acc, x0r * y0r + x0i * y0i + x1r * y1r + x1i * y1i);
  }
  block_reduce_store<256>(acc, d_part, blockIdx.x);
}

template <typename R>
__global__ void __launch_bounds__(256) k_inner(const typename C2<R>::T* __restrict__ a,
                                               const typename C2<R>::T* __restrict__ b, uint64_t N, double* d_part) {
  DD re{0, 0}, im{0, 0};
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    auto x = a[i];
    auto y = b[i];
    two_sum_acc(re, (double)x.x * y.x + (double)x.y * y.y);
    two_sum_acc(im, (double)x.x * y.y - (double)x.y * y.x);
  }
  block_reduce_store<256>(re, d_part, blockIdx.x);
  __syncthreads();
  block_reduce_store<256>(im, d_part, gridDim.x + blockIdx.x);
}

// Distance of a state a (complex64 or complex128) from a complex128 state b, d_i = a_i - b_i.
// Per block, as double-double partials: |d|^2, <b|d> (real, imaginary), |a|^2, |b|^2 and
// sum_i | |a_i|^2 - |b_i|^2 |, the last as |Re(d_i conj(a_i + b_i))| so that it does not
// cancel; and max_i |d_i|^2. 1 - F follows without cancellation from the identity
// <a|a><b|b> - |<b|a>|^2 = <b|b><d|d> - |<b|d>|^2.
template <typename R>
__global__ void __launch_bounds__(256) k_compare(const typename C2<R>::T* __restrict__ a,
                                                 const double2* __restrict__ b, uint64_t N, double* d_part,
                                                 double* d_max) {
  DD dd{0, 0}, re{0, 0}, im{0, 0}, na{0, 0}, nb{0, 0}, tv{0, 0};
  double mx = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    auto x = a[i];
    double2 y = b[i];
    double ar = (double)x.x, ai = (double)x.y;
    double dr = ar - y.x, di = ai - y.y;
    double d2 = dr * dr + di * di;
    two_sum_acc(dd, d2);
    two_sum_acc(re, y.x * dr + y.y * di);
    two_sum_acc(im, y.x * di - y.y * dr);
    two_sum_acc(na, ar * ar + ai * ai);
    two_sum_acc(nb, y.x * y.x + y.y * y.y);
    two_sum_acc(tv, fabs(dr * (ar + y.x) + di * (ai + y.y)));
    mx = fmax(mx, d2);
  }
  const DD acc[6] = {dd, re, im, na, nb, tv};
  for (int k = 0; k < 6; ++k) {
    block_reduce_store<256>(acc[k], d_part, k * gridDim.x + blockIdx.x);
    __syncthreads();
  }
  __shared__ double mred[8];
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) mred[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = mred[0];
    for (int w = 1; w < 8; ++w) m = fmax(m, mred[w]);
    d_max[blockIdx.x] = m;
  }
}

// Measurement of m distinct qubits without a trip to the host: k_marginal sums every outcome's
// probability (compensated FP64) and quantised probability (integers), k_measure_pick draws
// the outcome and k_collapse projects on it. Bound by the FP64 pipe: three instructions per
// probability, 16 of them summed exactly in fixed point (fixed_sum.cuh) before each TwoSum (20
// qubits, three measured: 56 us with a TwoSum per amplitude and an FP64 quantisation), and by
// launches: the host used to wait for the partial sums of every measurement (about 70 us each).
struct MeasuredBits {
  int m;
  int pos[16];   // the measured bits, ascending
  int rank[16];  // outcome bit of each
};
__device__ __forceinline__ uint64_t spread(uint64_t j, const MeasuredBits& f, uint32_t o) {
#pragma unroll 1
  for (int i = 0; i < f.m; ++i) {
    const int b = f.pos[i];
    const uint64_t lo = j & ((1ULL << b) - 1);
    j = ((j >> b) << (b + 1)) | ((uint64_t)((o >> f.rank[i]) & 1u) << b) | lo;
  }
  return j;
}

template <typename R>
__global__ void __launch_bounds__(256) k_marginal(const typename C2<R>::T* __restrict__ s, uint64_t work,
                                                  const MeasuredBits f, double* __restrict__ d_pm,
                                                  unsigned long long* __restrict__ d_qm) {
  const uint32_t o = blockIdx.y;
  DD acc{0, 0};
  unsigned long long qs = 0;
  for (uint64_t t = (uint64_t)blockIdx.x * 4096; t < work; t += (uint64_t)gridDim.x * 4096) {
    double v[16];
    uint32_t key = 0;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const uint64_t j = t + threadIdx.x + (uint64_t)r * 256;
      v[r] = j < work ? p_of<R>(s[spread(j, f, o)]) : 0.0;
      qs += quant(v[r]);
      key = max(key, qg_fix_key(v[r]));
    }
    const int E = qg_fix_exponent(key);
    int64_t h = 0, l = 0;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const qg_fixed x = qg_fix(v[r], E, 0);
      h += x.h;
      l += x.l;
    }
    two_sum_acc(acc, qg_fix_hi(h, E));
    acc.c = __dadd_rn(acc.c, qg_fix_lo(l, E));
  }
  const int slot = (int)(o * gridDim.x + blockIdx.x);
  block_reduce_store<256>(acc, d_pm, slot);
  __shared__ unsigned long long qred[8];
  for (int off = 16; off > 0; off >>= 1) qs += __shfl_down_sync(0xffffffffu, qs, off);
  if ((threadIdx.x & 31) == 0) qred[threadIdx.x >> 5] = qs;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; ++w) t += qred[w];
    d_qm[slot] = t;
  }
}

// One CTA. A warp folds each outcome's partials; the first warp then takes the first outcome
// whose cumulative quantised probability exceeds floor(draw T / 2^64) (the last one when T is
// 0), each lane over its share of the outcomes.
__global__ void __launch_bounds__(1024) k_measure_pick(const double* __restrict__ pm,
                                                       const unsigned long long* __restrict__ qm, int nbx,
                                                       const MeasuredBits f, uint64_t draw, double* __restrict__ P,
                                                       unsigned long long* __restrict__ Q, MeasurePick* out) {
  const int nout = 1 << f.m, lane = threadIdx.x & 31;
  for (int o = threadIdx.x >> 5; o < nout; o += 32) {
    DD a{0, 0};
    unsigned long long q = 0;
    for (int b = lane; b < nbx; b += 32) {
      const int slot = o * nbx + b;
      two_sum_acc(a, pm[2 * slot]);
      a.c = __dadd_rn(a.c, pm[2 * slot + 1]);
      q += qm[slot];
    }
    for (int d = 16; d > 0; d >>= 1) {
      DD w;
      w.s = __shfl_down_sync(0xffffffffu, a.s, d);
      w.c = __shfl_down_sync(0xffffffffu, a.c, d);
      a = dd_add(a, w);
      q += __shfl_down_sync(0xffffffffu, q, d);
    }
    if (lane == 0) {
      P[o] = __dadd_rn(a.s, a.c);
      Q[o] = q;
    }
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int per = (nout + 31) / 32, first = lane * per, last = min(nout, first + per);
  unsigned long long mine = 0;
  for (int o = first; o < last; ++o) mine += Q[o];
  unsigned long long incl = mine;
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
  }
  const unsigned long long T = __shfl_sync(0xffffffffu, incl, 31), u = __umul64hi(draw, T);
  const unsigned ballot = __ballot_sync(0xffffffffu, incl > u);
  const int owner = T > 0 ? __ffs((int)ballot) - 1 : 31;
  if (lane != owner) return;
  int sel = nout - 1;
  if (T > 0) {
    unsigned long long c = incl - mine;
    for (int o = first; o < last; ++o) {
      c += Q[o];
      if (c > u) {
        sel = o;
        break;
      }
    }
  }
  out->outcome = (uint64_t)sel;
  out->probability = P[sel];
  out->scale = P[sel] > 0 ? __ddiv_rn(1.0, __dsqrt_rn(P[sel])) : 1.0;
  uint64_t mask = 0, val = 0;
  for (int i = 0; i < f.m; ++i) {
    mask |= 1ULL << f.pos[i];
    if ((sel >> f.rank[i]) & 1) val |= 1ULL << f.pos[i];
  }
  out->mask = mask;
  out->val = val;
}

template <typename R>
__global__ void __launch_bounds__(256) k_collapse(typename C2<R>::T* __restrict__ s, uint64_t N,
                                                  const MeasurePick* __restrict__ pick) {
  using V = typename C2<R>::T;
  const uint64_t mask = pick->mask, val = pick->val;
  const R scale = (R)pick->scale;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
    V r;
    r.x = 0;
    r.y = 0;
    if ((i & mask) == val) {
      const V x = s[i];
      r.x = mul_(x.x, scale);
      r.y = mul_(x.y, scale);
    }
    s[i] = r;
  }
}

template <typename R>
__global__ void k_gather(const typename C2<R>::T* __restrict__ s, const uint64_t* __restrict__ idx, int64_t count,
                         double* __restrict__ out) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < count; j += (int64_t)gridDim.x * blockDim.x) {
    auto a = s[idx[j]];
    out[2 * j] = a.x;
    out[2 * j + 1] = a.y;
  }
}

template <typename R>
__global__ void k_density(const typename C2<R>::T* __restrict__ s, uint64_t N, double* __restrict__ rho) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < N * N; e += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t i = e / N, j = e % N;
    auto a = s[i];
    auto b = s[j];
    // a_i conj(a_j)
    rho[2 * e] = (double)a.x * b.x + (double)a.y * b.y;
    rho[2 * e + 1] = (double)a.y * b.x - (double)a.x * b.y;
  }
}

__global__ void k_set_one(void* s, int prec, uint64_t idx) {
  if (prec == QG_C64) reinterpret_cast<float2*>(s)[idx] = make_float2(1.f, 0.f);
  else reinterpret_cast<double2*>(s)[idx] = make_double2(1.0, 0.0);
}

__global__ void k_c128_to_c64(const double2* __restrict__ a, float2* __restrict__ b, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    double2 v = a[i];
    b[i] = make_float2((float)v.x, (float)v.y);
  }
}
__global__ void k_c64_to_c128(const float2* __restrict__ a, double2* __restrict__ b, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    float2 v = a[i];
    b[i] = make_double2(v.x, v.y);
  }
}

// ---------------------------------------------------------------------------
// Hierarchical sampler. Probabilities are quantised q_i = floor(p_i 2^62);
// chunk (32 amplitudes) and block (256 chunks) sums are exact integers, so the
// cumulative distribution does not depend on launch shape. A shot draws
// u = floor(r64 * T / 2^64) from Philox and takes the first i whose cumulative
// sum exceeds u: block by a search of the block prefix, then one of 16 groups of 16
// chunks, the chunk and the amplitude, each by a scan over lanes.
// ---------------------------------------------------------------------------
struct SampleGeom {
  uint64_t N;
  int ch;       // amplitudes per chunk (<= 32)
  int cpb;      // chunks per block (<= 256)
  uint64_t nb;  // blocks
  uint64_t nchunks;
};
SampleGeom sample_geom(int n) {
  SampleGeom g;
  g.N = 1ULL << n;
  g.ch = (int)(g.N < 32 ? g.N : 32);
  uint64_t nch = g.N / g.ch;
  g.cpb = (int)(nch < 256 ? nch : 256);
  g.nchunks = nch;
  g.nb = nch / g.cpb;
  return g;
}

// floor((re^2 + im^2) 2^62) of a complex64 amplitude, for parts below 2^-10, with eight
// instructions on the integer pipe (qg_quant62_sq_fast takes 29: it aligns both squares by
// variable shifts). With x' = |x| 2^41 and X = floor(x'), x'^2 = X^2 + (x' - X)(x' + X). X is a
// conversion, the squares are two wide multiply-adds, and the second term is zero from 2^-18
// on (x' is whole there); below, it comes from FP32 in units of z = x' 2^-23 cut off at 1,
// where zt = floor(z 2^23) 2^-23 is an addition of 1 that rounds to zero. z - zt is exact;
// z + zt, the product and the sum of both parts round to zero, so that
//   Sf = X^2 + Y^2 + floor(D) <= p 2^82 < Sf + 9 (per part 2 + 1, the sum 2, the floor 1),
// and Sf >> 20 is the value unless its fraction and the rounding of the FP64 sum (at most
// (Sf >> 52) + 4 units, see qg_quant62_fix) reach the next whole number. `worst` is the
// largest of fraction + (Sf >> 52) and `part` the largest magnitude (NaN stays NaN):
// the value holds when worst <= kWorstOk and part < 2^-10.
constexpr uint32_t kWorstOk = (1u << 20) - 16u;
__device__ __forceinline__ uint64_t quant62_wide(float re, float im, uint32_t& worst, float& part) {
  using u64 = unsigned long long;
  auto pk = [](float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
  };
  asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(part) : "f"(re), "f"(im));
  const uint32_t X = __float2uint_rz(fabsf(re) * 0x1p41f), Y = __float2uint_rz(fabsf(im) * 0x1p41f);
  const u64 z = pk(__saturatef(fabsf(re) * 0x1p18f), __saturatef(fabsf(im) * 0x1p18f));
  u64 zp, zt, f, g, d;
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(zp) : "l"(z), "l"(pk(1.f, 1.f)));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(zt) : "l"(zp), "l"(pk(-1.f, -1.f)));
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(f) : "l"(zp), "l"(pk(-0x1p46f, -0x1p46f)), "l"(pk(0x1p46f, 0x1p46f)));  // -zt 2^46
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(f) : "l"(z), "l"(pk(0x1p46f, 0x1p46f)));
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(g) : "l"(z), "l"(zt));
  asm("mul.rz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f), "l"(g));
  float d0, d1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d0), "=f"(d1) : "l"(d));
  const uint64_t s = (uint64_t)X * X + ((uint64_t)Y * Y + __float2uint_rz(__fadd_rz(d0, d1)));
  worst = max(worst, ((uint32_t)s & 0xFFFFFu) + (uint32_t)(s >> 52));
  return s >> 20;
}

// one CTA (256 threads = 8 warps) per sample block. Only integer sums are formed here:
// the FP64 total of the normalisation check is derived from them (k_samp_scan). A
// compensated FP64 reduction per chunk ran on the FP64 pipe (about 1/58 of the FP32
// rate on this part) and bound the whole sampler by it.
// Full blocks (256 chunks of 32 amplitudes: states of 13 qubits and more; every state the
// runtime allocates is aligned to 16 bytes and more): warp w takes the block's chunks 32w ..
// 32w + 31, four lanes to a chunk, with 16-byte loads, eight per lane in flight (one
// amplitude per lane and load for complex128, two for complex64). A lane adds up what it
// holds of a chunk before it exchanges anything: three exchanges per 32 chunks. (With a
// load spread over one or two whole chunks they were 15 for complex64 and 36 for complex128,
// of 8 instructions each.) Integer sums are associative: every chunk sum equals the
// lane-per-amplitude form's. The quantised probabilities come from fixed-point forms without
// an FP64 instruction (quant62_wide for complex64, qg_quant62_sq_fast for complex128), and,
// one vote per group of loads, from the FP64 expression where their guards fail; all give the
// same integers. Parts of 2^-10 or more fail, and since the probabilities sum to one, at most
// 2^20 amplitudes of a state have them. complex128 votes on the group's largest part first
// and sends such groups to the FP64 expression whole. Three CTAs per SM: 80 registers (ptxas
// otherwise picks 64 for complex128 and spills).
// complex64, 30 qubits: 1547 us, 82 % of the copy rate (1855 us bound by the integer pipe
// when the squares were aligned by variable shifts, 1994 us with 15 exchanges).
template <typename R>
__global__ void __launch_bounds__(256, 3) k_samp_sums(const typename C2<R>::T* __restrict__ s, SampleGeom g,
                                                   unsigned long long* __restrict__ csum,
                                                   unsigned long long* __restrict__ gsum,
                                                   unsigned long long* __restrict__ bsum) {
  using T = typename C2<R>::T;
  constexpr int A = 16 / (int)sizeof(T);  // amplitudes per 16-byte load
  constexpr int L = 4;                    // lanes per chunk
  constexpr int CPR = 32 / L;             // chunks per round of the warp
  constexpr int LOADS = 32 / (A * L);     // loads per lane and chunk
  constexpr int U = A == 2 ? 8 : 4;       // loads in flight per lane (8 spill for complex128)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ unsigned long long wq[8];
  for (uint64_t b = blockIdx.x; b < g.nb; b += gridDim.x) {
    unsigned long long bq = 0;
    if (g.cpb == 256) {
      const uint64_t c0 = b * 256 + (uint64_t)warp * 32;  // the warp's first chunk
      const uint4* src = reinterpret_cast<const uint4*>(s + (c0 + (uint64_t)(lane / L)) * 32) + lane % L;
      uint64_t w[L];  // round k: chunk CPR k + lane / L
#pragma unroll
      for (int k = 0; k < L; ++k) w[k] = 0;
#pragma unroll
      for (int i0 = 0; i0 < L * LOADS; i0 += U) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          v[u] = __ldg(src + (i0 + u) / LOADS * (CPR * 32 / A) + (i0 + u) % LOADS * L);
        uint64_t q[U];
        unsigned slow = 0;
        if constexpr (A == 2) {
          uint32_t worst = 0;
          float part = 0.f;
#pragma unroll
          for (int u = 0; u < U; ++u)
            q[u] = quant62_wide(__uint_as_float(v[u].x), __uint_as_float(v[u].y), worst, part) +
                   quant62_wide(__uint_as_float(v[u].z), __uint_as_float(v[u].w), worst, part);
          if (!(worst <= kWorstOk && part < 0x1p-10f)) slow = (1u << U) - 1;
        } else {
          bool big = false;
#pragma unroll
          for (int u = 0; u < U; ++u)  // high words: sign, exponent, top of the significand
            big |= max(v[u].y & 0x7FFFFFFFu, v[u].w & 0x7FFFFFFFu) >= (1013u << 20);
          slow = (1u << U) - 1;
          if (!__any_sync(0xffffffffu, big)) {
            slow = 0;
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const bool f = qg_quant62_sq_fast(__hiloint2double((int)v[u].y, (int)v[u].x),
                                                __hiloint2double((int)v[u].w, (int)v[u].z), &q[u]);
              slow |= (unsigned)!f << u;
            }
          }
        }
        if (__any_sync(0xffffffffu, slow)) {  // the FP64 expression
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (slow & (1u << u)) {
              if constexpr (A == 2) {
                const float2 x0 = make_float2(__uint_as_float(v[u].x), __uint_as_float(v[u].y));
                const float2 x1 = make_float2(__uint_as_float(v[u].z), __uint_as_float(v[u].w));
                uint64_t q0, q1;
                if (!qg_quant62_sq_fast(x0.x, x0.y, &q0)) q0 = quant(p_of<R>(x0));
                if (!qg_quant62_sq_fast(x1.x, x1.y, &q1)) q1 = quant(p_of<R>(x1));
                q[u] = q0 + q1;
              } else {
                const double2 x = make_double2(__hiloint2double((int)v[u].y, (int)v[u].x),
                                               __hiloint2double((int)v[u].w, (int)v[u].z));
                q[u] = quant(p_of<R>(x));
              }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) w[(i0 + u) / LOADS] += q[u];
      }
      // recursive halving (each step a lane sends the half of its partials it does not
      // keep): lane l ends with the sum of chunk CPR (l % L) + l / L
#pragma unroll
      for (int o = L / 2, K = L; o >= 1; o >>= 1, K >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < K / 2; ++i) {
          const uint64_t send = up ? w[i] : w[i + K / 2];
          const uint64_t keep = up ? w[i + K / 2] : w[i];
          w[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      csum[c0 + (uint64_t)(CPR * (lane % L) + lane / L)] = w[0];
      bq = w[0];
      // the sums of 16 chunks: the lanes of one value of bit 1
#pragma unroll
      for (int o : {1, 4, 8, 16}) bq += __shfl_xor_sync(0xffffffffu, bq, o);
      if ((lane & 29) == 0) gsum[c0 / 16 + (uint64_t)(lane >> 1)] = bq;
      bq += __shfl_xor_sync(0xffffffffu, bq, 2);
    } else {
      for (int c = warp; c < g.cpb; c += 8) {
        uint64_t chunk = b * g.cpb + c;
        unsigned long long q = 0;
        if (lane < g.ch) q = quant(p_of<R>(s[chunk * g.ch + lane]));
        for (int o = 16; o > 0; o >>= 1) q += __shfl_down_sync(0xffffffffu, q, o);
        if (lane == 0) {
          csum[chunk] = q;
          bq += q;
        }
      }
    }
    if (lane == 0) wq[warp] = bq;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t = 0;
      for (int w = 0; w < 8; ++w) t += wq[w];
      bsum[b] = t;
    }
    __syncthreads();
  }
}

// Exclusive prefix of block sums (bpre[nb] = T) and the FP64 total
// T 2^-62 + N 2^-63: every quantised probability lost less than one unit of
// 2^-62 to the floor, so the estimate is within N 2^-63 of sum p (2e-9 at 34
// qubits, well inside the 1e-8 normalisation tolerance). Latency-bound: a CTA takes 8192 sums,
// eight rows of 1024, through warp shuffles; with more than that (27 qubits and up) each CTA
// leaves its total in place of its first sum and k_samp_scan_add adds up those before it
// (30 qubits, 2^17 sums: 11 us; one CTA in 16 steps 93 us, 138 us with 16 consecutive sums
// per thread, whose loads and stores touch a line per lane, 228 us with a 1024-entry scan in
// shared memory per step).
constexpr int kScanRows = 8;
constexpr uint64_t kScanStep = 1024 * kScanRows;
__device__ __forceinline__ void scan_end(unsigned long long T, uint64_t n_amps, uint64_t nb,
                                         unsigned long long* bpre, double* total) {
  total[0] = (double)T * 0x1p-62 + (double)n_amps * 0x1p-63;
  bpre[nb] = T;
}
__global__ void __launch_bounds__(1024) k_samp_scan(unsigned long long* __restrict__ bsum, uint64_t nb,
                                                    uint64_t n_amps, unsigned long long* __restrict__ bpre,
                                                    double* __restrict__ total) {
  __shared__ unsigned long long wsum[kScanRows][32], wpre[kScanRows][32], rows[kScanRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t base = blockIdx.x * kScanStep + threadIdx.x;
  unsigned long long v[kScanRows], incl[kScanRows], carry = 0;
#pragma unroll
  for (int k = 0; k < kScanRows; ++k) {
    const uint64_t i = base + (uint64_t)k * 1024;
    incl[k] = v[k] = i < nb ? bsum[i] : 0ULL;
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
#pragma unroll
    for (int k = 0; k < kScanRows; ++k) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, incl[k], o);
      if (lane >= o) incl[k] += up;
    }
  if (lane == 31)
#pragma unroll
    for (int k = 0; k < kScanRows; ++k) wsum[k][warp] = incl[k];
  __syncthreads();
  if (warp < kScanRows) {  // warp w scans the warp sums of row w
    const unsigned long long x = wsum[warp][lane];
    unsigned long long s = x;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += up;
    }
    wpre[warp][lane] = s - x;
    if (lane == 31) rows[warp] = s;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kScanRows; ++k) {
    const uint64_t i = base + (uint64_t)k * 1024;
    if (i < nb) bpre[i] = carry + wpre[k][warp] + incl[k] - v[k];
    carry += rows[k];
  }
  if (threadIdx.x == 0) {
    if (gridDim.x == 1) scan_end(carry, n_amps, nb, bpre, total);
    else bsum[base] = carry;
  }
}
// CTA c adds the totals of the CTAs before it (nb = gridDim.x * kScanStep, 256 CTAs at most)
__global__ void __launch_bounds__(1024) k_samp_scan_add(const unsigned long long* __restrict__ bsum, uint64_t nb,
                                                        uint64_t n_amps, unsigned long long* __restrict__ bpre,
                                                        double* __restrict__ total) {
  __shared__ unsigned long long part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long before = threadIdx.x < blockIdx.x ? bsum[(uint64_t)threadIdx.x * kScanStep] : 0ULL;
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (lane == 0) part[warp] = before;
  __syncthreads();
  before = part[lane];
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  const uint64_t base = blockIdx.x * kScanStep + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kScanRows; ++k) bpre[base + (uint64_t)k * 1024] += before;
  if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1)
    scan_end(before + bsum[(uint64_t)blockIdx.x * kScanStep], n_amps, nb, bpre, total);
}

// States below 13 qubits (one block of at most 128 chunks): one warp per shot, up to four
// consecutive chunk sums per lane.
template <typename R>
__global__ void __launch_bounds__(256) k_samp_resolve_small(const typename C2<R>::T* __restrict__ s, SampleGeom g,
                                                            const unsigned long long* __restrict__ csum,
                                                            const unsigned long long* __restrict__ bpre,
                                                            uint64_t shots, uint64_t seed,
                                                            uint64_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const uint64_t stride = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned long long T = bpre[g.nb];
  const int per = (g.cpb + 31) / 32;
  for (uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < shots; k += stride) {
    if (T == 0) {
      if (lane == 0) out[k] = 0;
      continue;
    }
    const unsigned long long r = __umul64hi(draw64(seed, k, 0u), T);
    unsigned long long loc[4], mine = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      loc[c] = c < per && lane * per + c < g.cpb ? csum[lane * per + c] : 0ULL;
      mine += loc[c];
    }
    unsigned long long incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    // the owner's first chunk whose cumulative sum exceeds r (the last one where sums of infinite
    // amplitudes wrapped)
    const int owner = __ffs((int)(__ballot_sync(0xffffffffu, incl > r) | 0x80000000u)) - 1;
    unsigned long long before = incl - mine;
    int chunk = lane * per;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (chunk == lane * per + c && c < per - 1 && before + loc[c] <= r) {
        before += loc[c];
        ++chunk;
      }
    chunk = __shfl_sync(0xffffffffu, chunk < g.cpb ? chunk : g.cpb - 1, owner);
    before = __shfl_sync(0xffffffffu, before, owner);
    unsigned long long qi = lane < g.ch ? quant(p_of<R>(s[chunk * g.ch + lane])) : 0ULL;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, qi, o);
      if (lane >= o) qi += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, lane < g.ch && before + qi > r);
    const int pick = hit ? __ffs((int)hit) - 1 : g.ch - 1;
    if (lane == 0) out[k] = (uint64_t)chunk * g.ch + pick;
  }
}

// Half a warp per shot, `batch` (1..16) shots one after the other with their draws computed
// side by side. The block is found 16 ways at a time among (up to) 4096 evenly spaced
// prefixes that each CTA keeps in shared memory, every level of that tree packed, and from
// there 32 ways in bpre, where 2^17 blocks leave 32 consecutive prefixes. The chunk comes
// from the sums of 16 chunks and then the chunks' own, the amplitude from a scan of the
// chunk, all contiguous. Bound by instruction issue and the latency of scattered reads (30
// qubits, 10^6 shots: 977 us with a binary search and one Philox draw per lane and shot, 727 us
// with 32-way steps through bpre, a line per lane, and all 256 chunk sums of the block read,
// 441 us with a warp per shot, 283 us).
constexpr int kTop = 4096;
template <typename R>
__global__ void __launch_bounds__(512, 3) k_samp_resolve(const typename C2<R>::T* __restrict__ s, SampleGeom g,
                                                         const unsigned long long* __restrict__ csum,
                                                         const unsigned long long* __restrict__ gsum,
                                                         const unsigned long long* __restrict__ bpre, uint64_t shots,
                                                         uint64_t seed, int batch, uint64_t* __restrict__ out) {
  // top[i] = bpre at the end of the i-th of `tops` equal runs of blocks; mid and head hold
  // every 16th entry of the level below (entries past the end read T)
  __shared__ unsigned long long top[kTop], mid[kTop / 16], head[16];
  const int lane = threadIdx.x & 15, half = threadIdx.x & 16;
  const unsigned long long T = bpre[g.nb];
  const int tops = (int)(g.nb < kTop ? g.nb : kTop);  // a power of two, as g.nb
  const uint64_t run = g.nb / (uint64_t)tops;
  for (int i = threadIdx.x; i < tops; i += blockDim.x) top[i] = bpre[(uint64_t)(i + 1) * run];
  __syncthreads();
  if (tops > 16) {
    if (threadIdx.x < kTop / 16) mid[threadIdx.x] = threadIdx.x < tops / 16 ? top[16 * threadIdx.x + 15] : T;
    if (threadIdx.x < 16) head[threadIdx.x] = threadIdx.x < tops / 256 ? top[256 * threadIdx.x + 255] : T;
    __syncthreads();
  }
  auto vote = [&](bool p) { return (__ballot_sync(0xffffffffu, p) >> half) & 0xffffu; };
  // the last lane without a hit: sums that wrapped (infinite amplitudes) stay in bounds
  auto first_of = [&](bool p) { return __ffs((int)(vote(p) | 0x8000u)) - 1; };
  auto scan = [&](unsigned long long v) {  // inclusive, over the half-warp
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, v, o, 16);
      if (lane >= o) v += up;
    }
    return v;
  };
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t at = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 2 * batch; at < shots;
       at += warps * 2 * batch) {
    const uint64_t first = at + (half ? (uint64_t)batch : 0);
    const int cnt = first >= shots ? 0 : (int)(shots - first < (uint64_t)batch ? shots - first : (uint64_t)batch);
    const int most = (int)(shots - at < (uint64_t)batch ? shots - at : (uint64_t)batch);  // the lower half's count
    unsigned long long draw = 0, picked = 0;
    if (lane < cnt) draw = __umul64hi(draw64(seed, first + lane, 0u), T);
    if (T != 0)
      for (int q = 0; q < most; ++q) {  // past its count the upper half looks for 0
        const unsigned long long u = __shfl_sync(0xffffffffu, draw, q, 16);
        // block: first b with bpre[b + 1] > u; bpre[nb] = T > u, so every vote has a winner
        int t = 0;
        if (tops > 256) t = first_of(head[lane] > u);
        if (tops > 16) t = 16 * t + first_of(mid[16 * t + lane] > u);
        t = 16 * t + first_of(lane >= tops || top[16 * t + lane] > u);
        uint64_t b = (uint64_t)t * run, len = run;
        while (len > 1) {  // 32 ways, two per lane; len is a power of two
          const uint64_t step = (len + 31) >> 5, to = (uint64_t)(2 * lane + 1) * step;
          const unsigned odd = vote(bpre[b + (to < len ? to : len)] > u);
          const int l = first_of(bpre[b + (to + step < len ? to + step : len)] > u);
          b += (uint64_t)(2 * l + 1 - (int)((odd >> l) & 1u)) * step;
          len = step;
        }
        unsigned long long r = u - bpre[b];
        // one of 16 groups of 16 chunks, then the chunk: two lines of memory instead of 2 KB
        uint64_t chunk = b * 16;
#pragma unroll
        for (int level = 0; level < 2; ++level) {
          const unsigned long long mine = (level == 0 ? gsum : csum)[chunk + lane], incl = scan(mine);
          const int owner = first_of(incl > r);
          r -= __shfl_sync(0xffffffffu, incl - mine, owner, 16);
          chunk += owner;
          if (level == 0) chunk *= 16;
        }
        // its 32 amplitudes, two per lane: the fixed-point path as in k_samp_sums, the FP64
        // expression past its guard
        unsigned long long qa[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const typename C2<R>::T a = s[chunk * 32 + 2 * lane + e];
          uint64_t x;
          if (!qg_quant62_sq_fast(a.x, a.y, &x)) x = quant(p_of<R>(a));
          qa[e] = x;
        }
        const unsigned long long incl = scan(qa[0] + qa[1]);
        const unsigned even = vote(incl - qa[1] > r);
        const int l = first_of(incl > r);
        if (lane == q) picked = chunk * 32 + 2 * l + 1 - ((even >> l) & 1u);
      }
    if (lane < cnt) out[first + lane] = picked;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
unsigned long long kernel_launch_count() { return g_launches.load(); }
void count_launch(int k) { counted(k); }

int reduce_blocks_for(int n) {
  uint64_t N = 1ULL << n;
  uint64_t b = (N + 255) / 256;
  if (b > (uint64_t)kSMs * 4) b = (uint64_t)kSMs * 4;
  return (int)(b < 1 ? 1 : b);
}

cudaError_t launch_set_basis(void* s, int precision, int n, uint64_t idx, cudaStream_t st) {
  size_t bytes = (precision == QG_C64 ? 8ULL : 16ULL) << n;
  cudaError_t e = cudaMemsetAsync(s, 0, bytes, st);
  if (e != cudaSuccess) return e;
  k_set_one<<<1, 1, 0, st>>>(s, precision, idx);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_plain_op(void* s, int precision, int n, const GOp& op, cudaStream_t st) {
  return precision == QG_C64 ? plain_op_t<float>(s, n, op, st) : plain_op_t<double>(s, n, op, st);
}

cudaError_t launch_c128_to_c64(const double* src, float* dst, uint64_t count, cudaStream_t st) {
  k_c128_to_c64<<<grid_for(count, 256), 256, 0, st>>>((const double2*)src, (float2*)dst, count);
  counted();
  return cudaGetLastError();
}
cudaError_t launch_c64_to_c128(const float* src, double* dst, uint64_t count, cudaStream_t st) {
  k_c64_to_c128<<<grid_for(count, 256), 256, 0, st>>>((const float2*)src, (double2*)dst, count);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_probabilities(const void* s, int precision, int n, double* d_p, cudaStream_t st) {
  uint64_t N = 1ULL << n;
  if (precision == QG_C64) k_probs<float><<<grid_for(N, 256), 256, 0, st>>>((const float2*)s, N, d_p);
  else k_probs<double><<<grid_for(N, 256), 256, 0, st>>>((const double2*)s, N, d_p);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_norm2(const void* s, int precision, int n, double* d_part, int nblocks, cudaStream_t st) {
  uint64_t N = 1ULL << n;
  if (precision == QG_C64) k_norm2<float><<<nblocks, 256, 0, st>>>((const float2*)s, N, d_part);
  else k_norm2<double><<<nblocks, 256, 0, st>>>((const double2*)s, N, d_part);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_expect_1q(const void* s, int precision, int n, int bit, const double* o8, double* d_part,
                             int nblocks, cudaStream_t st) {
  uint64_t N = 1ULL << n;
  Mat<double> o = to_mat<double>(o8);
  if (precision == QG_C64) k_expect1q<float><<<nblocks, 256, 0, st>>>((const float2*)s, N, bit, o, d_part);
  else k_expect1q<double><<<nblocks, 256, 0, st>>>((const double2*)s, N, bit, o, d_part);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_inner(const void* a, const void* b, int precision, int n, double* d_part, int nblocks,
                         cudaStream_t st) {
  uint64_t N = 1ULL << n;
  if (precision == QG_C64) k_inner<float><<<nblocks, 256, 0, st>>>((const float2*)a, (const float2*)b, N, d_part);
  else k_inner<double><<<nblocks, 256, 0, st>>>((const double2*)a, (const double2*)b, N, d_part);
  counted();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Noisy trajectories: end of a shot. The Kraus operators were applied without
// renormalisation, so each distinct trajectory state is first scaled by 1 / ||a||
// (state.clj:524-551: every amplitude times (/ 1.0 norm)), one CTA per state. Then
// every shot draws one outcome from its state the way the shot sampler draws:
// quantised probabilities q_i = floor(p_i 2^62), their integer total T,
// u = floor(r64 T / 2^64) and the first i whose inclusive prefix sum exceeds u, one
// CTA per shot. Each thread owns a contiguous chunk of the state; the chunk sums are
// scanned in shared memory and the chunk that holds u is walked by its thread.
// ---------------------------------------------------------------------------
// Bound by the FP64 pipe: a shuffle step of the compensated sum costs about 20 FP64
// instructions per warp, so a state gets as many warps as leave 32 amplitudes to each lane
// (launch_traj_normalise; 7,700 states of 10 qubits: 362 us with 256 threads each, 215 us).
template <typename R>
__global__ void __launch_bounds__(256) k_traj_normalise(void* const* __restrict__ states, int n,
                                                        double* __restrict__ norm2) {
  using T = typename C2<R>::T;
  T* s = reinterpret_cast<T*>(states[blockIdx.x]);
  const uint64_t N = 1ULL << n;
  __shared__ DD red[8];
  __shared__ double scale_sh;
  DD acc{0, 0};
#pragma unroll 8
  for (uint64_t i = threadIdx.x; i < N; i += blockDim.x) two_sum_acc(acc, p_of<R>(s[i]));
  for (int o = 16; o > 0; o >>= 1) {
    DD w;
    w.s = __shfl_down_sync(0xffffffffu, acc.s, o);
    w.c = __shfl_down_sync(0xffffffffu, acc.c, o);
    acc = dd_add(acc, w);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    DD t = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = dd_add(t, red[w]);
    const double nn = t.s + t.c;
    norm2[blockIdx.x] = nn;
    scale_sh = nn > 0 ? 1.0 / sqrt(nn) : 0.0;
  }
  __syncthreads();
  const double sc = scale_sh;
  for (uint64_t i = threadIdx.x; i < N; i += blockDim.x) {
    T a = s[i];
    a.x = (R)((double)a.x * sc);
    a.y = (R)((double)a.y * sc);
    s[i] = a;
  }
}

template <typename R>
__global__ void __launch_bounds__(256) k_traj_sample(void* const* __restrict__ states,
                                                     const int32_t* __restrict__ state_of, int n, int shift,
                                                     uint64_t seed, uint64_t traj0, uint32_t stream,
                                                     uint64_t* __restrict__ out) {
  using T = typename C2<R>::T;
  const T* s = reinterpret_cast<const T*>(states[state_of[blockIdx.x]]);
  const uint64_t N = 1ULL << n;
  const uint64_t chunk = (N + blockDim.x - 1) / blockDim.x;
  const uint64_t lo = min(N, (uint64_t)threadIdx.x * chunk), hi = min(N, lo + chunk);
  __shared__ unsigned long long pre[256];
  unsigned long long q = 0;
  for (uint64_t i = lo; i < hi; ++i) q += quant(p_of<R>(s[i]));
  pre[threadIdx.x] = q;
  __syncthreads();
  for (unsigned o = 1; o < blockDim.x; o <<= 1) {  // inclusive scan of the chunk sums
    const unsigned long long add = threadIdx.x >= o ? pre[threadIdx.x - o] : 0ULL;
    __syncthreads();
    pre[threadIdx.x] += add;
    __syncthreads();
  }
  const unsigned long long total = pre[blockDim.x - 1];
  if (total == 0) {
    if (threadIdx.x == 0) out[blockIdx.x] = 0;
    return;
  }
  const unsigned long long u = __umul64hi(draw64(seed, traj0 + blockIdx.x, stream), total);
  const unsigned long long before = pre[threadIdx.x] - q;
  if (u >= before && u < pre[threadIdx.x]) {
    unsigned long long c = before;
    for (uint64_t i = lo; i < hi; ++i) {
      c += quant(p_of<R>(s[i]));
      if (c > u) {
        out[blockIdx.x] = i >> shift;
        break;
      }
    }
  }
}

cudaError_t launch_traj_normalise(int precision, void* const* d_states, int nstates, int n, double* d_norm2,
                                  cudaStream_t st) {
  if (nstates < 1) return cudaSuccess;
  const int threads = n >= 13 ? 256 : n <= 10 ? 32 : 32 << (n - 10);
  if (precision == QG_C64) k_traj_normalise<float><<<nstates, threads, 0, st>>>(d_states, n, d_norm2);
  else k_traj_normalise<double><<<nstates, threads, 0, st>>>(d_states, n, d_norm2);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_traj_sample(int precision, void* const* d_states, const int32_t* d_state_of, int nshots, int n,
                               int shift, uint64_t seed, uint64_t traj0, uint32_t stream, uint64_t* d_out,
                               cudaStream_t st) {
  if (nshots < 1) return cudaSuccess;
  if (precision == QG_C64)
    k_traj_sample<float><<<nshots, 256, 0, st>>>(d_states, d_state_of, n, shift, seed, traj0, stream, d_out);
  else
    k_traj_sample<double><<<nshots, 256, 0, st>>>(d_states, d_state_of, n, shift, seed, traj0, stream, d_out);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_compare(const void* a, int precision, const void* b, int n, double* d_part, double* d_max,
                           int nblocks, cudaStream_t st) {
  uint64_t N = 1ULL << n;
  if (precision == QG_C64)
    k_compare<float><<<nblocks, 256, 0, st>>>((const float2*)a, (const double2*)b, N, d_part, d_max);
  else
    k_compare<double><<<nblocks, 256, 0, st>>>((const double2*)a, (const double2*)b, N, d_part, d_max);
  counted();
  return cudaGetLastError();
}

// scratch: measure_scratch_bytes(m); *pick is device memory
static int measure_chunks(int n, int m) {
  const uint64_t work = (1ULL << n) >> m;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((work + 4095) / 4096, 1024u >> m));
}
size_t measure_scratch_bytes(int n, int m) {
  const size_t slots = (size_t)measure_chunks(n, m) << m;
  return slots * (2 * sizeof(double) + sizeof(unsigned long long)) +
         ((size_t)1 << m) * (sizeof(double) + sizeof(unsigned long long));
}
cudaError_t launch_measure(void* s, int precision, int n, const int* bits, int m, uint64_t draw, void* d_scratch,
                           MeasurePick* d_pick, cudaStream_t st) {
  MeasuredBits f;
  f.m = m;
  int at = 0;
  for (int b = 0; b < n; ++b)
    for (int k = 0; k < m; ++k)
      if (bits[k] == b) {
        f.pos[at] = b;
        f.rank[at++] = k;
      }
  const uint64_t N = 1ULL << n, work = N >> m;
  const int nbx = measure_chunks(n, m);
  const size_t slots = (size_t)nbx << m;
  double* pm = reinterpret_cast<double*>(d_scratch);
  unsigned long long* qm = reinterpret_cast<unsigned long long*>(pm + 2 * slots);
  double* P = reinterpret_cast<double*>(qm + slots);
  unsigned long long* Q = reinterpret_cast<unsigned long long*>(P + ((size_t)1 << m));
  const dim3 grid((unsigned)nbx, 1u << m);
  if (precision == QG_C64) k_marginal<float><<<grid, 256, 0, st>>>((const float2*)s, work, f, pm, qm);
  else k_marginal<double><<<grid, 256, 0, st>>>((const double2*)s, work, f, pm, qm);
  k_measure_pick<<<1, 1024, 0, st>>>(pm, qm, nbx, f, draw, P, Q, d_pick);
  if (precision == QG_C64) k_collapse<float><<<grid_for(N, 256), 256, 0, st>>>((float2*)s, N, d_pick);
  else k_collapse<double><<<grid_for(N, 256), 256, 0, st>>>((double2*)s, N, d_pick);
  counted(3);
  return cudaGetLastError();
}

cudaError_t launch_gather(const void* s, int precision, const uint64_t* d_idx, int64_t count, double* d_out,
                          cudaStream_t st) {
  int g = grid_for((uint64_t)count, 256);
  if (precision == QG_C64) k_gather<float><<<g, 256, 0, st>>>((const float2*)s, d_idx, count, d_out);
  else k_gather<double><<<g, 256, 0, st>>>((const double2*)s, d_idx, count, d_out);
  counted();
  return cudaGetLastError();
}

cudaError_t launch_density(const void* s, int precision, int n, double* d_rho, cudaStream_t st) {
  uint64_t N = 1ULL << n;
  int g = grid_for(N * N, 256);
  if (precision == QG_C64) k_density<float><<<g, 256, 0, st>>>((const float2*)s, N, d_rho);
  else k_density<double><<<g, 256, 0, st>>>((const double2*)s, N, d_rho);
  counted();
  return cudaGetLastError();
}

size_t sampler_scratch_bytes(int n, uint64_t shots) {
  (void)shots;
  return sampler_scratch_bytes_at(n);  // the layout of sample_geom(n) below
}

cudaError_t launch_sample(const void* s, int precision, int n, uint64_t shots, uint64_t seed, void* d_scratch,
                          uint64_t* d_outcomes, double* d_total, cudaStream_t st) {
  SampleGeom g = sample_geom(n);
  unsigned long long* csum = (unsigned long long*)d_scratch;
  unsigned long long* gsum = csum + g.nchunks;
  unsigned long long* bsum = gsum + 16 * g.nb;
  unsigned long long* bpre = bsum + g.nb;
  int grid = (int)(g.nb < (uint64_t)kSMs * 8 ? g.nb : (uint64_t)kSMs * 8);
  if (precision == QG_C64)
    k_samp_sums<float><<<grid, 256, 0, st>>>((const float2*)s, g, csum, gsum, bsum);
  else
    k_samp_sums<double><<<grid, 256, 0, st>>>((const double2*)s, g, csum, gsum, bsum);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const unsigned scans = (unsigned)((g.nb + kScanStep - 1) / kScanStep);
  k_samp_scan<<<scans, 1024, 0, st>>>(bsum, g.nb, g.N, bpre, d_total);
  if (scans > 1) k_samp_scan_add<<<scans, 1024, 0, st>>>(bsum, g.nb, g.N, bpre, d_total);
  e = cudaGetLastError();
  counted(scans > 1 ? 3 : 2);
  if (e != cudaSuccess || shots == 0) return e;
  if (g.cpb < 256) {
    const unsigned blocks = (unsigned)std::min<uint64_t>((shots + 7) / 8, (uint64_t)kSMs * 8);
    if (precision == QG_C64)
      k_samp_resolve_small<float><<<blocks, 256, 0, st>>>((const float2*)s, g, csum, bpre, shots, seed, d_outcomes);
    else
      k_samp_resolve_small<double><<<blocks, 256, 0, st>>>((const double2*)s, g, csum, bpre, shots, seed, d_outcomes);
  } else {
    // equal batches of at most 16 in whole rounds of the grid (three CTAs of 32 half-warps per SM)
    const uint64_t most = (uint64_t)kSMs * 3 * 32, round = 16 * most;
    const uint64_t rounds = std::max<uint64_t>(1, (shots + round - 1) / round);
    const int batch = (int)std::max<uint64_t>(1, (shots + rounds * most - 1) / (rounds * most));
    const uint64_t halves = (shots + batch - 1) / batch;
    const unsigned blocks = (unsigned)std::min<uint64_t>((halves + 31) / 32, (uint64_t)kSMs * 3);
    if (precision == QG_C64)
      k_samp_resolve<float><<<blocks, 512, 0, st>>>((const float2*)s, g, csum, gsum, bpre, shots, seed, batch,
                                                    d_outcomes);
    else
      k_samp_resolve<double><<<blocks, 512, 0, st>>>((const double2*)s, g, csum, gsum, bpre, shots, seed, batch,
                                                     d_outcomes);
  }
  counted();
  return cudaGetLastError();
}

}  // namespace qg
