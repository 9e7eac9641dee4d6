// Device prelude of the specialised pass kernels (pass_kernels.cpp).
//
// A tiled pass (one HBM read and write of the state that applies a run of
// gates, see tile.cu) is compiled into its own kernel: the generated code
// names every gate with its matrix entries as literals, its register slots and
// its conditions, so the gate run is straight-line code with no op dispatch.
// This file holds what every such kernel shares:
//   - run_pass<P>: the tile loop (cp.async double-buffered 16-byte copies into
//     an XOR-swizzled shared-memory tile, P::body applied to the tile, coalesced
//     16-byte stores), with the pass geometry supplied by P;
//   - the complex arithmetic of the two policies the generator emits:
//       complex128 as double-float pairs (hi + lo floats, about 48 bits) on the
//       FP32 pipes, with error-free products (FMA) and sums (TwoSum), real and
//       imaginary part together in packed instructions; results are left unnormalised (the pair (s, t) of a rounded sum and its
//       collected error) and renormalised by the generated code after a few
//       operations on a register and before it is stored;
//       complex64 in FP32 with FMA contraction.
// It is compiled by NVRTC together with df64.cuh; it includes no system header.
#pragma once

#include "df64.cuh"

// Powers of w = exp(2 pi i / 2^30) in three tables of 1024 (w^(a 2^20), w^(b 2^10),
// w^c), double-float (re.hi, re.lo, im.hi, im.lo); filled by the host after the
// module is loaded. Runs of phases that are all such powers (the controlled
// phases of a QFT) add integer exponents and look the product up here.
__device__ float4 qgp_roots[3072];

namespace qgp {

using qg::dfc;
typedef unsigned long long u64;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// XOR swizzle of the shared-memory tile (16-byte units, 8 per 128-byte row; 8-byte
// amplitudes move in 16-byte pairs). Every index bit above the row's three unit bits is
// folded onto one of them, so all bits fall into three classes (position mod 3), and any
// lanes whose three low bits carry one index bit of each class touch eight different
// units: the generator picks the lanes' bits that way in every layout (thread_map).
template <int E>
__device__ __forceinline__ int swz(int l) {
  if (E == 16) return l ^ (((l >> 3) ^ (l >> 6) ^ (l >> 9) ^ (l >> 12)) & 7);
  return l ^ ((((l >> 4) ^ (l >> 7) ^ (l >> 10)) & 7) << 1);
}

// ---------------------------------------------------------------------------
// Packed FP32 (f32x2): one instruction works on two floats. It has the same rate per float as
// the scalar form (a probe on GB300: 123 of 128 floats per clock and SM either way) for half
// the issue slots, and the double-float passes are bound by issue and by the latency of their
// chains, not by the FP32 lanes: the two halves of an operand are the real and the imaginary
// part, which every gate treats alike. Each lane does the operations of the scalar form
// (products, FMA error terms, TwoSum) in the same order, so results are the same bits.
// There is no packed negation: differences and negated constants take its place. ptxas contracts
// a packed product into the packed sums that use it when nothing else does (unlike the scalar
// .rn forms), which would break a TwoSum of it: mul2 is for products whose FMA error term uses
// the rounded product too, and for exact ones; mul2_rn rounds lane by lane.
// ---------------------------------------------------------------------------
__device__ __forceinline__ u64 pk(float a, float b) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpk(u64 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
  u64 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 mul2_rn(u64 a, u64 b) {
  float ax, ay, bx, by;
  unpk(a, ax, ay);
  unpk(b, bx, by);
  return pk(__fmul_rn(ax, bx), __fmul_rn(ay, by));
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a complex double-float as two operands: leading floats (re, im), trailing floats (re, im)
struct cp {
  u64 h, l;
};
__device__ __forceinline__ cp pack(const dfc& x) { return cp{pk(x.rh, x.ih), pk(x.rl, x.il)}; }
__device__ __forceinline__ cp pack_swapped(const dfc& x) { return cp{pk(x.ih, x.rh), pk(x.il, x.rl)}; }
__device__ __forceinline__ dfc unpack(const cp& x) {
  dfc y;
  unpk(x.h, y.rh, y.ih);
  unpk(x.l, y.rl, y.il);
  return y;
}
// a constant pair per lane (re lane: ah + al, im lane: bh + bl) and its negation
struct kp {
  u64 h, l, nh, nl;
};
__device__ __forceinline__ kp konst(float ah, float al, float bh, float bl) {
  return kp{pk(ah, bh), pk(al, bl), pk(-ah, -bh), pk(-al, -bl)};
}
__device__ __forceinline__ kp konst(float h, float l) { return konst(h, l, h, l); }

// Knuth's TwoSum: s = fl(a + b), e = (a + b) - s exactly.
__device__ __forceinline__ void tsum(u64 a, u64 b, u64& s, u64& e) {
  s = add2(a, b);
  const u64 bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
// the same for a - b
__device__ __forceinline__ void tdiff(u64 a, u64 b, u64& s, u64& e) {
  s = sub2(a, b);
  const u64 bb = sub2(s, a);
  e = sub2(sub2(a, sub2(s, bb)), add2(b, bb));
}
// k * x: p = fl(kh * xh) and n = -(its exact error plus the cross terms kh * xl and kl * xh)
template <bool KL>
__device__ __forceinline__ void tprod(const kp& k, const cp& x, u64& p, u64& n) {
  p = mul2(k.h, x.h);
  n = fma2(k.nh, x.h, p);
  n = fma2(k.nh, x.l, n);
  if (KL) n = fma2(k.nl, x.h, n);
}
// the same with the signs exchanged: n = -fl(kh * xh), e = +(error and cross terms)
template <bool KL>
__device__ __forceinline__ void tprod_neg(const kp& k, const cp& x, u64& n, u64& e) {
  n = mul2(k.nh, x.h);
  e = fma2(k.h, x.h, n);
  e = fma2(k.h, x.l, e);
  if (KL) e = fma2(k.l, x.h, e);
}
// k * x
template <bool KL>
__device__ __forceinline__ cp prod(const kp& k, const cp& x) {
  u64 n, e;
  tprod_neg<KL>(k, x, n, e);
  return cp{mul2_rn(k.h, x.h), e};
}
// a*x + b*y, unnormalised
template <bool AL, bool BL>
__device__ __forceinline__ cp dot2(const kp& a, const cp& x, const kp& b, const cp& y) {
  u64 p1, n1, p2, n2, s, err;
  tprod<AL>(a, x, p1, n1);
  tprod<BL>(b, y, p2, n2);
  tsum(p1, p2, s, err);
  return cp{s, sub2(err, add2(n1, n2))};
}
// x + y and x - y, unnormalised
__device__ __forceinline__ cp sum(const cp& x, const cp& y) {
  u64 s, err;
  tsum(x.h, y.h, s, err);
  return cp{s, add2(add2(x.l, y.l), err)};
}
__device__ __forceinline__ cp diff(const cp& x, const cp& y) {
  u64 s, err;
  tdiff(x.h, y.h, s, err);
  return cp{s, add2(sub2(x.l, y.l), err)};
}
// x + k*y, unnormalised
template <bool KL>
__device__ __forceinline__ cp axpy(const kp& k, const cp& x, const cp& y) {
  u64 n, e, s, err;
  tprod_neg<KL>(k, y, n, e);
  tdiff(x.h, n, s, err);
  return cp{s, add2(add2(x.l, e), err)};
}
// k*y - x, unnormalised
template <bool KL>
__device__ __forceinline__ cp axmy(const kp& k, const cp& x, const cp& y) {
  u64 p, n, s, err;
  tprod<KL>(k, y, p, n);
  tdiff(p, x.h, s, err);
  return cp{s, sub2(err, add2(x.l, n))};
}
// Fast2Sum: bring the collected error back under the leading float. The
// generated code applies it to a register after a few products (and before a
// register goes to shared memory): left to grow, the low float random-walks to
// a sizeable fraction of the high one and its roundings no longer average out
// (the state's norm then drifts by ~1e-11 over a thousand gates).
__device__ __forceinline__ cp fast2(const cp& x) {
  const u64 s = add2(x.h, x.l);
  return cp{s, sub2(x.l, sub2(s, x.h))};
}

// ---- complex double-float ------------------------------------------------
struct DF {
  typedef dfc V;
  static constexpr int E = 16;
  static __device__ __forceinline__ V ld_work(const unsigned char* b, int pos) {
    const float4 v = reinterpret_cast<const float4*>(b)[pos];
    return dfc{v.x, v.y, v.z, v.w};
  }
  static __device__ __forceinline__ void st_work(unsigned char* b, int pos, const V& v) {
    reinterpret_cast<float4*>(b)[pos] = make_float4(v.rh, v.ih, v.rl, v.il);
  }
  static __device__ __forceinline__ V ld_doubles(const unsigned char* b, int pos) {
    return qg::load_dfc(reinterpret_cast<const double2*>(b)[pos]);
  }
  // normalised pairs (|l| <= ulp(h)/2) for the conversion to IEEE doubles
  static __device__ __forceinline__ void st_doubles(unsigned char* b, int pos, const V& v) {
    const cp x = pack(v);
    cp y;
    tsum(x.h, x.l, y.h, y.l);
    reinterpret_cast<double2*>(b)[pos] = qg::store_dfc(unpack(y));
  }
  static __device__ __forceinline__ V renorm(const V& v) { return unpack(fast2(pack(v))); }
  static __device__ __forceinline__ V neg(const V& x) { return dfc{-x.rh, -x.ih, -x.rl, -x.il}; }
  static __device__ __forceinline__ V mul_i(const V& x) { return dfc{-x.ih, x.rh, -x.il, x.rl}; }
  static __device__ __forceinline__ V mul_mi(const V& x) { return dfc{x.ih, -x.rh, x.il, -x.rl}; }
};

// (gr + i gi) * x: re = gr xr + (-gi) xi, im = gr xi + gi xr
template <bool RL, bool IL>
__device__ __forceinline__ cp df_cmul_p(float grh, float grl, float gih, float gil, const dfc& x) {
  return dot2<RL, IL>(konst(grh, grl), pack(x), konst(-gih, -gil, gih, gil), pack_swapped(x));
}
template <bool RL, bool IL>
__device__ __forceinline__ dfc df_cmul(float grh, float grl, float gih, float gil, const dfc& x) {
  return unpack(df_cmul_p<RL, IL>(grh, grl, gih, gil, x));
}
// (a + i a) x (NEG = false) or (a - i a) x (NEG = true), a a constant pair: x + i x or
// x - i x first, then one product each (a T-gate phase)
template <bool AL, bool NEG>
__device__ __forceinline__ dfc df_cmul_diag(float ah, float al, const dfc& x) {
  return unpack(prod<AL>(konst(ah, al), sum(pack(x), pack(NEG ? DF::mul_mi(x) : DF::mul_i(x)))));
}
// y = a*x0 + b*x1 for complex constants a, b (8 floats: a.re h/l, a.im h/l, b.re h/l, b.im h/l)
__device__ __forceinline__ dfc df_row(float arh, float arl, float aih, float ail, float brh, float brl, float bih,
                                      float bil, const dfc& x0, const dfc& x1) {
  return unpack(sum(df_cmul_p<true, true>(arh, arl, aih, ail, x0), df_cmul_p<true, true>(brh, brl, bih, bil, x1)));
}
// real 2x2 [[a, b], [c, d]]
template <bool AL, bool BL, bool CL, bool DL>
__device__ __forceinline__ void df_real(float ah, float al, float bh, float bl, float ch, float cl, float dh, float dl,
                                        dfc& x0, dfc& x1) {
  const cp u = pack(x0), v = pack(x1);
  x0 = unpack(dot2<AL, BL>(konst(ah, al), u, konst(bh, bl), v));
  x1 = unpack(dot2<CL, DL>(konst(ch, cl), u, konst(dh, dl), v));
}
// [[c, c], [c, -c]] (Hadamard-shaped): the sum and difference first, one product each
template <bool CL>
__device__ __forceinline__ void df_hadamard(float ch, float cl, dfc& x0, dfc& x1) {
  const cp u = pack(x0), v = pack(x1);
  const kp c = konst(ch, cl);
  x0 = unpack(prod<CL>(c, sum(u, v)));
  x1 = unpack(prod<CL>(c, diff(u, v)));
}
// [[1, 1], [1, -1]]: a Hadamard whose 1/sqrt 2 is applied later with the global factors
__device__ __forceinline__ void df_sumdiff(dfc& x0, dfc& x1) {
  const cp u = pack(x0), v = pack(x1);
  x0 = unpack(sum(u, v));
  x1 = unpack(diff(u, v));
}
// [[1, b], [c, S]] (S = +-1): a real rotation with its diagonal factored out
template <bool BL, bool CL, bool NEG>
__device__ __forceinline__ void df_realunit(float bh, float bl, float ch, float cl, dfc& x0, dfc& x1) {
  const cp u = pack(x0), v = pack(x1);
  x0 = unpack(axpy<BL>(konst(bh, bl), u, v));
  x1 = unpack(NEG ? axmy<CL>(konst(ch, cl), v, u) : axpy<CL>(konst(ch, cl), v, u));
}
// [[1, i b], [i c, 1]]: an RX-shaped rotation with its diagonal factored out
template <bool BL, bool CL>
__device__ __forceinline__ void df_rxunit(float bh, float bl, float ch, float cl, dfc& x0, dfc& x1) {
  const cp u = pack(x0), us = pack_swapped(x0), v = pack(x1), vs = pack_swapped(x1);
  x0 = unpack(axpy<BL>(konst(-bh, -bl, bh, bl), u, vs));
  x1 = unpack(axpy<CL>(konst(-ch, -cl, ch, cl), v, us));
}
// x * w^T, the chunks the run needs selected at compile time
template <bool A, bool B, bool C>
__device__ __forceinline__ dfc df_root_mul_impl(unsigned T, const dfc& x) {
  dfc g = dfc{1.0f, 0.0f, 0.0f, 0.0f};
  bool have = false;
  if (A) {
    const float4 v = qgp_roots[(T >> 20) & 1023u];
    g = dfc{v.x, v.z, v.y, v.w};
    have = true;
  }
  if (B) {
    const float4 v = qgp_roots[1024 + ((T >> 10) & 1023u)];
    g = have ? df_cmul<true, true>(v.x, v.y, v.z, v.w, g) : dfc{v.x, v.z, v.y, v.w};
    have = true;
  }
  if (C) {
    const float4 v = qgp_roots[2048 + (T & 1023u)];
    g = have ? df_cmul<true, true>(v.x, v.y, v.z, v.w, g) : dfc{v.x, v.z, v.y, v.w};
  }
  return df_cmul<true, true>(g.rh, g.rl, g.ih, g.il, x);
}
// x times a power of two (exact)
__device__ __forceinline__ dfc df_pow2(float c, const dfc& x) {
  const cp v = pack(x);
  const u64 k = pk(c, c);
  return unpack(cp{mul2(k, v.h), mul2(k, v.l)});
}
// [[a, i b], [i c, d]] with a, b, c, d real (RX-shaped)
template <bool AL, bool BL, bool CL, bool DL>
__device__ __forceinline__ void df_rxlike(float ah, float al, float bh, float bl, float ch, float cl, float dh, float dl,
                                          dfc& x0, dfc& x1) {
  const cp u = pack(x0), us = pack_swapped(x0), v = pack(x1), vs = pack_swapped(x1);
  x0 = unpack(dot2<AL, BL>(konst(ah, al), u, konst(-bh, -bl, bh, bl), vs));
  x1 = unpack(dot2<DL, CL>(konst(dh, dl), v, konst(-ch, -cl, ch, cl), us));
}

// ---- complex64 -------------------------------------------------------------
struct F32 {
  typedef float2 V;
  static constexpr int E = 8;
  static __device__ __forceinline__ V ld_work(const unsigned char* b, int pos) {
    return reinterpret_cast<const float2*>(b)[pos];
  }
  static __device__ __forceinline__ void st_work(unsigned char* b, int pos, const V& v) {
    reinterpret_cast<float2*>(b)[pos] = v;
  }
  // two registers in the 16-byte slot pair (pos, pos + 1), pos even
  static __device__ __forceinline__ void ld_pair(const unsigned char* b, int pos, V& a, V& c) {
    const float4 v = *reinterpret_cast<const float4*>(b + pos * 8);
    a = make_float2(v.x, v.y);
    c = make_float2(v.z, v.w);
  }
  static __device__ __forceinline__ void st_pair(unsigned char* b, int pos, const V& a, const V& c) {
    *reinterpret_cast<float4*>(b + pos * 8) = make_float4(a.x, a.y, c.x, c.y);
  }
  static __device__ __forceinline__ V neg(const V& x) { return make_float2(-x.x, -x.y); }
  static __device__ __forceinline__ V mul_i(const V& x) { return make_float2(-x.y, x.x); }
  static __device__ __forceinline__ V mul_mi(const V& x) { return make_float2(x.y, -x.x); }
};
__device__ __forceinline__ float2 f_cmul(float gr, float gi, float2 x) {
  return make_float2(fmaf(gr, x.x, -(gi * x.y)), fmaf(gr, x.y, gi * x.x));
}
__device__ __forceinline__ float2 f_row(float ar, float ai, float br, float bi, float2 x0, float2 x1) {
  return make_float2(fmaf(ar, x0.x, fmaf(-ai, x0.y, fmaf(br, x1.x, -(bi * x1.y)))),
                     fmaf(ar, x0.y, fmaf(ai, x0.x, fmaf(br, x1.y, bi * x1.x))));
}
__device__ __forceinline__ void f_real(float a, float b, float c, float d, float2& x0, float2& x1) {
  const float2 y0 = make_float2(fmaf(a, x0.x, b * x1.x), fmaf(a, x0.y, b * x1.y));
  const float2 y1 = make_float2(fmaf(c, x0.x, d * x1.x), fmaf(c, x0.y, d * x1.y));
  x0 = y0;
  x1 = y1;
}
__device__ __forceinline__ void f_hadamard(float c, float2& x0, float2& x1) {
  const float2 y0 = make_float2(c * (x0.x + x1.x), c * (x0.y + x1.y));
  const float2 y1 = make_float2(c * (x0.x - x1.x), c * (x0.y - x1.y));
  x0 = y0;
  x1 = y1;
}
__device__ __forceinline__ void f_sumdiff(float2& x0, float2& x1) {
  const float2 y0 = make_float2(x0.x + x1.x, x0.y + x1.y);
  const float2 y1 = make_float2(x0.x - x1.x, x0.y - x1.y);
  x0 = y0;
  x1 = y1;
}
__device__ __forceinline__ float2 f_pow2(float c, float2 x) { return make_float2(x.x * c, x.y * c); }
template <bool A, bool B, bool C>
__device__ __forceinline__ float2 f_root_mul_impl(unsigned T, float2 x) {
  float2 g = make_float2(1.0f, 0.0f);
  if (A) {
    const float4 v = qgp_roots[(T >> 20) & 1023u];
    g = f_cmul(v.x, v.z, g);
  }
  if (B) {
    const float4 v = qgp_roots[1024 + ((T >> 10) & 1023u)];
    g = f_cmul(v.x, v.z, g);
  }
  if (C) {
    const float4 v = qgp_roots[2048 + (T & 1023u)];
    g = f_cmul(v.x, v.z, g);
  }
  return f_cmul(g.x, g.y, x);
}
template <bool NEG>
__device__ __forceinline__ void f_realunit(float b, float c, float2& x0, float2& x1) {
  const float2 y0 = make_float2(fmaf(b, x1.x, x0.x), fmaf(b, x1.y, x0.y));
  const float2 y1 = NEG ? make_float2(fmaf(c, x0.x, -x1.x), fmaf(c, x0.y, -x1.y))
                        : make_float2(fmaf(c, x0.x, x1.x), fmaf(c, x0.y, x1.y));
  x0 = y0;
  x1 = y1;
}
__device__ __forceinline__ void f_rxunit(float b, float c, float2& x0, float2& x1) {
  const float2 y0 = make_float2(fmaf(-b, x1.y, x0.x), fmaf(b, x1.x, x0.y));
  const float2 y1 = make_float2(fmaf(-c, x0.y, x1.x), fmaf(c, x0.x, x1.y));
  x0 = y0;
  x1 = y1;
}
__device__ __forceinline__ void f_rxlike(float a, float b, float c, float d, float2& x0, float2& x1) {
  const float2 y0 = make_float2(fmaf(a, x0.x, -(b * x1.y)), fmaf(a, x0.y, b * x1.x));
  const float2 y1 = make_float2(fmaf(d, x1.x, -(c * x0.y)), fmaf(c, x0.x, d * x1.y));
  x0 = y0;
  x1 = y1;
}

// ---------------------------------------------------------------------------
// The tile loop. P supplies: E (bytes per amplitude in HBM), K_BITS, KLOW,
// R_BITS (each of the 2^(K_BITS - R_BITS) threads holds 2^R_BITS amplitudes),
// BUFS (1: one tile buffer, the SM's other CTAs overlap their copies with this
// one's arithmetic; 2 or 3: the next one or two tiles are prefetched), LM
// (mask of the local bit positions), hioff(h) (HBM offset, in amplitudes, of the
// h-th 2^KLOW-amplitude run of a tile), tile_base(t) (first amplitude of tile t)
// and body(buf, base, cs) (the gate run on the tile in shared memory; it ends
// with a barrier; cs holds the matrix entries when they come from a table). Each
// CTA walks a contiguous range of tiles.
// ---------------------------------------------------------------------------
template <class P>
__device__ __forceinline__ void run_pass(unsigned char* __restrict__ state, u64 ntiles) {
  constexpr int E = P::E, K = 1 << P::K_BITS, T = K >> P::R_BITS, PER = 16 / E, CPT = (K * E / 16) / T;
  extern __shared__ __align__(128) unsigned char smem[];
  u64 goff[CPT];
  unsigned soff[CPT];
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int l = ((int)threadIdx.x + i * T) * PER;
    goff[i] = ((u64)(l & ((1 << P::KLOW) - 1)) | P::hioff(l >> P::KLOW)) * E;
    soff[i] = (unsigned)swz<E>(l) * E;
  }
  const u64 w0 = ntiles * blockIdx.x / gridDim.x, w1 = ntiles * (blockIdx.x + 1) / gridDim.x;
  if (w0 >= w1) return;
  u64 base = P::tile_base(w0);
  if (P::BUFS == 1) {
    for (u64 t = w0; t < w1; ++t) {
#pragma unroll
      for (int i = 0; i < CPT; ++i) cp_async16(smem + soff[i], state + base * E + goff[i]);
      cp_commit();
      cp_wait<0>();
      __syncthreads();
      P::body(smem, base, nullptr);
#pragma unroll
      for (int i = 0; i < CPT; ++i)
        *reinterpret_cast<uint4*>(state + base * E + goff[i]) = *reinterpret_cast<const uint4*>(smem + soff[i]);
      __syncthreads();  // the buffer is refilled by the next tile
      base = ((base | P::LM) + 1) & ~P::LM;
    }
    return;
  }
  // a ring of BUFS buffers: the next BUFS - 1 tiles are in flight while one is worked
  // on; one copy group is committed per tile (empty ones past the range), so waiting
  // for all but the newest BUFS - 1 groups waits for the current tile
  u64 pb = base, pt = w0;
#pragma unroll
  for (int q = 0; q < P::BUFS - 1; ++q) {
    if (pt < w1) {
#pragma unroll
      for (int i = 0; i < CPT; ++i) cp_async16(smem + q * (K * E) + soff[i], state + pb * E + goff[i]);
      pb = ((pb | P::LM) + 1) & ~P::LM;
      ++pt;
    }
    cp_commit();
  }
  int cb = 0, nbuf = P::BUFS - 1;  // buffer of the current tile, of the next prefetch
  for (u64 t = w0; t < w1; ++t) {
    unsigned char* cur = smem + cb * (K * E);
    if (pt < w1) {
#pragma unroll
      for (int i = 0; i < CPT; ++i) cp_async16(smem + nbuf * (K * E) + soff[i], state + pb * E + goff[i]);
      pb = ((pb | P::LM) + 1) & ~P::LM;
      ++pt;
    }
    cp_commit();
    cp_wait<P::BUFS - 1>();
    __syncthreads();
    P::body(cur, base, nullptr);
#pragma unroll
    for (int i = 0; i < CPT; ++i)
      *reinterpret_cast<uint4*>(state + base * E + goff[i]) = *reinterpret_cast<const uint4*>(cur + soff[i]);
    __syncthreads();  // this buffer is refilled by the next prefetch
    base = ((base | P::LM) + 1) & ~P::LM;
    nbuf = cb;
    cb = cb + 1 == P::BUFS ? 0 : cb + 1;
  }
}

// The same pass over many states of one structure (a parameter sweep): work
// items are (state, tile) pairs; a CTA walks a contiguous range [w0, w1) of them
// and, whenever it reaches a new state, stages that state's matrix entries (ncoef
// floats at coefs + state * ncoef) into shared memory after the tile buffers.
template <class P>
__device__ __forceinline__ void run_pass_range(unsigned char* const* __restrict__ states,
                                               const float* __restrict__ coefs, int ncoef, u64 ntiles, u64 w0,
                                               u64 w1) {
  constexpr int E = P::E, K = 1 << P::K_BITS, T = K >> P::R_BITS, PER = 16 / E, CPT = (K * E / 16) / T;
  extern __shared__ __align__(128) unsigned char smem[];
  float* cs = reinterpret_cast<float*>(smem + P::BUFS * K * E);
  u64 goff[CPT];
  unsigned soff[CPT];
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int l = ((int)threadIdx.x + i * T) * PER;
    goff[i] = ((u64)(l & ((1 << P::KLOW) - 1)) | P::hioff(l >> P::KLOW)) * E;
    soff[i] = (unsigned)swz<E>(l) * E;
  }
  for (u64 w = w0; w < w1;) {
    const int si = (int)(w / ntiles);
    const u64 t0 = w - (u64)si * ntiles;
    const u64 t1 = (ntiles - t0 < w1 - w) ? ntiles : t0 + (w1 - w);
    unsigned char* state = states[si];
    __syncthreads();  // the previous state's readers of cs are done
    for (int q = (int)threadIdx.x; q < ncoef; q += T) cs[q] = coefs[(u64)si * ncoef + q];
    u64 base = P::tile_base(t0);
    // the ring of run_pass (one buffer: the next tile is loaded after the store)
    u64 pb = base, pt = t0;
#pragma unroll
    for (int q = 0; q < (P::BUFS > 1 ? P::BUFS - 1 : 1); ++q) {
      if (pt < t1) {
#pragma unroll
        for (int i = 0; i < CPT; ++i) cp_async16(smem + q * (K * E) + soff[i], state + pb * E + goff[i]);
        pb = ((pb | P::LM) + 1) & ~P::LM;
        ++pt;
      }
      cp_commit();
    }
    int cb = 0, nbuf = P::BUFS > 1 ? P::BUFS - 1 : 0;
    for (u64 t = t0; t < t1; ++t) {
      unsigned char* cur = smem + cb * (K * E);
      if (P::BUFS > 1) {
        if (pt < t1) {
#pragma unroll
          for (int i = 0; i < CPT; ++i) cp_async16(smem + nbuf * (K * E) + soff[i], state + pb * E + goff[i]);
          pb = ((pb | P::LM) + 1) & ~P::LM;
          ++pt;
        }
        cp_commit();
        cp_wait<(P::BUFS > 1 ? P::BUFS - 1 : 0)>();
      } else {
        cp_wait<0>();
      }
      __syncthreads();
      P::body(cur, base, cs);
#pragma unroll
      for (int i = 0; i < CPT; ++i)
        *reinterpret_cast<uint4*>(state + base * E + goff[i]) = *reinterpret_cast<const uint4*>(cur + soff[i]);
      __syncthreads();  // the buffer is refilled by a later tile
      if (P::BUFS == 1 && pt < t1) {
#pragma unroll
        for (int i = 0; i < CPT; ++i) cp_async16(smem + soff[i], state + pb * E + goff[i]);
        pb = ((pb | P::LM) + 1) & ~P::LM;
        ++pt;
        cp_commit();
      }
      base = ((base | P::LM) + 1) & ~P::LM;
      if (P::BUFS > 1) {
        nbuf = cb;
        cb = cb + 1 == P::BUFS ? 0 : cb + 1;
      }
    }
    w += t1 - t0;
  }
}

// One launch per pass over all states of a group: CTA b takes its share of the items.
template <class P>
__device__ __forceinline__ void run_pass_batch(unsigned char* const* __restrict__ states,
                                               const float* __restrict__ coefs, int ncoef, u64 ntiles, int nstates) {
  const u64 W = ntiles * (u64)nstates;
  run_pass_range<P>(states, coefs, ncoef, ntiles, W * blockIdx.x / gridDim.x, W * (blockIdx.x + 1) / gridDim.x);
}

// Sweeps of several sizes: one launch per pass level runs the pass of that level of
// every group (qubit count) that has one. Each CTA takes an equal share of every
// group's (state, tile) items, group after group, as if each group had its own launch
// of the same grid: a group of many small states spreads its state switches (each one
// stages that state's coefficients and cannot prefetch across states) over all CTAs.
struct GroupLevel {
  unsigned char* const* states;
  const float* coefs;  // this pass's rows: ncoef floats per state
  int ncoef, nstates;
  u64 ntiles, item0, items;
};
template <class P>
__device__ __forceinline__ void run_group_share(const GroupLevel& d) {
  const u64 a = d.items * blockIdx.x / gridDim.x, b = d.items * (blockIdx.x + 1) / gridDim.x;
  if (a < b) run_pass_range<P>(d.states, d.coefs, d.ncoef, d.ntiles, a, b);
}

}  // namespace qgp
