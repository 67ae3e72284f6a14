// gl_gf61.cuh -- exact arithmetic in GF(q^2), q = 2^61 - 1, for the integer form of an
// iteration (gl_int_kernels.cu).
//
// GB300 issues FP64 at 2 lanes per clock and SM, 32-bit integer work at 64: the radix-8
// butterfly of the line DFTs takes 4640 sub-partition cycles per warp in FP64 and 1130 in
// this field (both measured from registers, twiddles from shared memory).  The products of
// an iteration are integers below 2^60, so their residues mod q determine them, without
// round-off.
//
// Why q = 2^61 - 1 and its quadratic extension (i^2 = -1; -1 is a non-residue):
//  * reduction is a shift and an add (2^61 = 1);
//  * 2 has order 61, so for every N not divisible by 61 the IBDWT weight 2^(r/N) is
//    2^(r N^-1 mod 61), a rotation by 0..60 bits;
//  * the group has roots of unity of every order 2^a 3^b 5^c 7^d with a <= 62, b, c <= 2,
//    d <= 1; sqrt(1/2) = 2^30, so the radix-8 constants are rotations too;
//  * x -> x^q is complex conjugation, so a transform of real words packed in pairs splits
//    as over the complex numbers (with k and q k mod M in place of k and M - k).
//
// Values are signed 64-bit and only partly reduced.  Write R for "at most 2^60 + 2^35 in
// magnitude", what red() and the products return; 3R < 2^62 is what a product accepts.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#ifndef GL_HD
#define GL_HD __host__ __device__ __forceinline__
#endif

namespace gl {
namespace gf {

constexpr uint64_t kQ = (1ull << 61) - 1;

struct __align__(16) g2 {
  int64_t re, im;
};

// A constant c of the field as c0 + c1 2^31, |c0| <= 2^30, |c1| <= 2^29, and a pair (c, d)
// for c + i d: the form in which every table holds its twiddles.
struct Limbs {
  int c0, c1;
};

GL_HD uint32_t lo32(uint64_t x) { return (uint32_t)x; }
GL_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
#ifdef __CUDA_ARCH__
// a b + c, 32 x 32 -> 64 bits (inline PTX: the compiler otherwise splits some of these
// into a product and a separate 64-bit addition)
GL_HD uint64_t mad_s(int a, int b, uint64_t c) {
  uint64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
GL_HD uint64_t mad_u(uint32_t a, uint32_t b, uint64_t c) {
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
GL_HD uint64_t pack(uint32_t l, uint32_t h) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(l), "r"(h));
  return r;
}
GL_HD uint32_t funnel(uint32_t l, uint32_t h, int s) { return __funnelshift_r(l, h, s); }
#else
GL_HD uint64_t mad_s(int a, int b, uint64_t c) { return (uint64_t)((int64_t)a * b) + c; }
GL_HD uint64_t mad_u(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }
GL_HD uint64_t pack(uint32_t l, uint32_t h) { return ((uint64_t)h << 32) | l; }
GL_HD uint32_t funnel(uint32_t l, uint32_t h, int s) { return (uint32_t)((((uint64_t)h << 32) | l) >> s); }
#endif

// x reduced to [-2^60 - 4, 2^60 + 3], |x| < 2^63 - 2^60
GL_HD int64_t red(int64_t x) {
  const int hi = (int)hi32((uint64_t)x);
  const int h = (hi + (1 << 28)) >> 29;  // x = h 2^61 + a balanced remainder
  return (int64_t)mad_s(h, 1, pack(lo32((uint64_t)x), (uint32_t)(hi - h * (1 << 29))));
}

// The accumulators of a product start at these values, so that they stay positive; the
// first is 4 q, the second 4 q + 2^29, whose 2^29 (weight 2^31) the balancing takes back.
constexpr uint64_t kAccLo = (1ull << 63) - 4, kAccMid = (1ull << 63) - 4 + (1ull << 29);

// lo + mid 2^31 for biased accumulators, reduced to R
GL_HD int64_t fold(uint64_t lo, uint64_t mid) {
  const uint64_t t = mad_u(hi32(lo), 2u, mid);  // lo = low word + (high word) 2 2^31
  const uint64_t th = pack(funnel(lo32(t), hi32(t), 30), hi32(t) >> 30);  // t = th 2^30 + tl, 2^61 = 1
  return (int64_t)(mad_u(lo32(t) & 0x3fffffffu, 1u << 31, th + lo32(lo)) - (1ull << 60));
}

// the two 31-bit limbs of a value below 2^62 in magnitude: x = a0 + a1 2^31, 0 <= a0
GL_HD int limb0(int64_t x) { return (int)(lo32((uint64_t)x) & 0x7fffffffu); }
GL_HD int limb1(int64_t x) { return (int)funnel(lo32((uint64_t)x), hi32((uint64_t)x), 31); }

// x w, |re|, |im| < 2^62; accumulators: |lo| <= 2 (2^61 + 2^61), |mid| <= 2 (2^60 + 2^61)
GL_HD g2 cmul(g2 x, int4 w) {
  const int a0 = limb0(x.re), a1 = limb1(x.re), b0 = limb0(x.im), b1 = limb1(x.im);
  const int c2 = w.y * 2, d2 = w.w * 2;
  const int n0 = -w.z, n1 = -w.w, n2 = -d2;
  g2 r;
  {
    const uint64_t l = mad_s(b1, n2, mad_s(b0, n0, mad_s(a1, c2, mad_s(a0, w.x, kAccLo))));
    const uint64_t m = mad_s(b1, n0, mad_s(b0, n1, mad_s(a1, w.x, mad_s(a0, w.y, kAccMid))));
    r.re = fold(l, m);
  }
  {
    const uint64_t l = mad_s(b1, c2, mad_s(b0, w.x, mad_s(a1, d2, mad_s(a0, w.z, kAccLo))));
    const uint64_t m = mad_s(b1, w.x, mad_s(b0, w.y, mad_s(a1, w.z, mad_s(a0, w.w, kAccMid))));
    r.im = fold(l, m);
  }
  return r;
}
// x c, |x| < 2^62
GL_HD int64_t rmul(int64_t x, Limbs c) {
  const int a0 = limb0(x), a1 = limb1(x);
  return fold(mad_s(a1, 2 * c.c1, mad_s(a0, c.c0, kAccLo)), mad_s(a1, c.c0, mad_s(a0, c.c1, kAccMid)));
}
// x c + y d, |x|, |y| < 2^62
GL_HD int64_t rdot(int64_t x, Limbs c, int64_t y, Limbs d) {
  const int a0 = limb0(x), a1 = limb1(x), b0 = limb0(y), b1 = limb1(y);
  return fold(mad_s(b1, 2 * d.c1, mad_s(b0, d.c0, mad_s(a1, 2 * c.c1, mad_s(a0, c.c0, kAccLo)))),
              mad_s(b1, d.c0, mad_s(b0, d.c1, mad_s(a1, c.c0, mad_s(a0, c.c1, kAccMid)))));
}
// x y, |x| < 2^62, y within R
GL_HD int64_t vmul(int64_t x, int64_t y) { return rmul(x, Limbs{limb0(y), limb1(y)}); }

// x 2^30, |result| <= 2^61 + 2^33
GL_HD int64_t rot30(int64_t x) {
  const int lo = (int)lo32((uint64_t)x);
  const int xh = (int)hi32((uint64_t)x) + (int)((uint32_t)lo >> 31);
  return (int64_t)mad_s(lo, 1 << 30, mad_s(xh, 2, 0));
}

GL_HD g2 add(g2 a, g2 b) { return g2{a.re + b.re, a.im + b.im}; }
GL_HD g2 sub(g2 a, g2 b) { return g2{a.re - b.re, a.im - b.im}; }
GL_HD g2 red(g2 a) { return g2{red(a.re), red(a.im)}; }
// a + S i b, a - S i b
template <int S>
GL_HD g2 addi(g2 a, g2 b) {
  return S < 0 ? g2{a.re + b.im, a.im - b.re} : g2{a.re - b.im, a.im + b.re};
}
template <int S>
GL_HD g2 subi(g2 a, g2 b) {
  return addi<-S>(a, b);
}

// Compile-time powers in GF(q) for the constants of the odd radices.
constexpr uint64_t mulq(uint64_t a, uint64_t b) {
  const unsigned __int128 p = (unsigned __int128)a * b;
  const uint64_t s = (uint64_t)(p & kQ) + (uint64_t)(p >> 61);
  return s >= kQ ? s - kQ : s;
}
constexpr uint64_t powq(uint64_t a, uint64_t e) {
  uint64_t r = 1;
  for (; e; e >>= 1) {
    if (e & 1) r = mulq(r, a);
    a = mulq(a, a);
  }
  return r;
}
constexpr uint64_t kGen = 37;  // a primitive root mod q
static_assert(powq(kGen, (kQ - 1) / 2) == kQ - 1 && powq(kGen, (kQ - 1) / 3) != 1 &&
                  powq(kGen, (kQ - 1) / 5) != 1 && powq(kGen, (kQ - 1) / 7) != 1,
              "the roots of odd order come from this generator");
constexpr uint64_t kHalf = 1ull << 60;
// primitive root of odd order r used throughout (host tables and butterflies)
constexpr uint64_t root_odd(uint64_t r) { return powq(kGen, (kQ - 1) / r); }
constexpr Limbs limbs(uint64_t c) {
  int64_t v = c > (kQ >> 1) ? (int64_t)c - (int64_t)kQ : (int64_t)c;
  int64_t l = v & 0x7fffffff;
  if (l >= (1 << 30)) l -= (int64_t)1 << 31;
  return Limbs{(int)l, (int)((v - l) / ((int64_t)1 << 31))};
}
// (w^j + w^-j)/2 and (w^j - w^-j)/2 for w = root_odd(r)
constexpr Limbs half_sum(uint64_t r, uint64_t j) {
  const uint64_t w = root_odd(r);
  uint64_t s = powq(w, j) + powq(w, r - j);
  return limbs(mulq(s >= kQ ? s - kQ : s, kHalf));
}
constexpr Limbs half_dif(uint64_t r, uint64_t j) {
  const uint64_t w = root_odd(r);
  const uint64_t a = powq(w, j), b = powq(w, r - j);
  return limbs(mulq(a >= b ? a - b : a + kQ - b, kHalf));
}

constexpr Limbs neg(Limbs a) { return Limbs{-a.c0, -a.c1}; }
constexpr Limbs kW3f = limbs(root_odd(3)), kW3i = limbs(powq(root_odd(3), 2));
constexpr Limbs k5c1 = half_sum(5, 1), k5c2 = half_sum(5, 2), k5s1 = half_dif(5, 1), k5s2 = half_dif(5, 2);
constexpr Limbs k5n1 = neg(k5s1);
constexpr Limbs k7c1 = half_sum(7, 1), k7c2 = half_sum(7, 2), k7c3 = half_sum(7, 3);
constexpr Limbs k7s1 = half_dif(7, 1), k7s2 = half_dif(7, 2), k7s3 = half_dif(7, 3);
constexpr Limbs k7n1 = neg(k7s1), k7n3 = neg(k7s3);

// ---------------------------------------------------------------------------
// Small DFTs, y_k = sum_n x_n w^(nk); S = -1 forward (w of order 4 is -i, of order 8
// 2^30 (1 - i)), S = +1 inverse.  Inputs within R, outputs within 3R.
// ---------------------------------------------------------------------------
template <int S>
GL_HD void dft2(g2* x) {
  const g2 a = x[0], b = x[1];
  x[0] = add(a, b);
  x[1] = sub(a, b);
}

template <int S>
GL_HD void dft4(g2* x) {
  const g2 s = add(x[0], x[2]), d = sub(x[0], x[2]);
  const g2 t = red(add(x[1], x[3])), u = red(sub(x[1], x[3]));
  x[0] = add(s, t);
  x[2] = sub(s, t);
  x[1] = addi<S>(d, u);
  x[3] = subi<S>(d, u);
}

// the even or odd half of a radix-8 butterfly: DFT_4 of a, b, c, d, reduced
template <int S>
GL_HD void dft4_red(g2& a, g2& b, g2& c, g2& d) {
  const g2 s = add(a, c), t = add(b, d), u = sub(a, c), v = sub(b, d);
  a = red(add(s, t));
  c = red(sub(s, t));
  b = red(addi<S>(u, v));
  d = red(subi<S>(u, v));
}
// x[0..7] = even DFT_4 (e0, e1, e2, e3) and odd DFT_4 (o0, o1, o2, o3), interleaved; combined
template <int S>
GL_HD void dft8_join(g2* x) {
  // w8 = (1 + S i) 2^30, w8^3 = (-1 + S i) 2^30
  const g2 o1 = x[3], o3 = x[7];
  const g2 t1 = S < 0 ? g2{rot30(o1.re + o1.im), rot30(o1.im - o1.re)}
                      : g2{rot30(o1.re - o1.im), rot30(o1.im + o1.re)};
  const g2 t3 = S < 0 ? g2{rot30(o3.im - o3.re), rot30(-o3.im - o3.re)}
                      : g2{rot30(-o3.re - o3.im), rot30(o3.re - o3.im)};
  const g2 e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6], o0 = x[1], o2 = x[5];
  x[0] = add(e0, o0);
  x[4] = sub(e0, o0);
  x[2] = addi<S>(e2, o2);
  x[6] = subi<S>(e2, o2);
  x[1] = add(e1, t1);
  x[5] = sub(e1, t1);
  x[3] = add(e3, t3);
  x[7] = sub(e3, t3);
}

// w = root_odd(3), a scalar of GF(q): w^2 = -1 - w, so
// y1 = x0 - x2 + w (x1 - x2), y2 = x0 - x1 - w (x1 - x2)
template <int S>
GL_HD void dft3(g2* x) {
  constexpr Limbs w = S < 0 ? kW3f : kW3i;
  const g2 d = sub(x[1], x[2]);
  const g2 t = g2{rmul(d.re, w), rmul(d.im, w)};
  const g2 y1 = add(sub(x[0], x[2]), t), y2 = sub(sub(x[0], x[1]), t);
  x[0] = add(x[0], add(x[1], x[2]));
  x[1] = y1;
  x[2] = y2;
}

// Roots of odd order are scalars, so real and imaginary parts transform separately (which
// also halves the values live at once).
template <int S>
GL_HD void dft5_part(int64_t& x0, int64_t& x1, int64_t& x2, int64_t& x3, int64_t& x4) {
  constexpr Limbs c1 = k5c1, c2 = k5c2, s1 = k5s1, s2 = k5s2, m1 = k5n1;
  const int64_t t1 = x1 + x4, t2 = x2 + x3, d1 = x1 - x4, d2 = x2 - x3;
  const int64_t a1 = x0 + rdot(t1, c1, t2, c2), a2 = x0 + rdot(t1, c2, t2, c1);
  const int64_t b1 = rdot(d1, s1, d2, s2), b2 = rdot(d1, s2, d2, m1);
  x0 += red(t1 + t2);
  x1 = S < 0 ? a1 + b1 : a1 - b1;
  x4 = S < 0 ? a1 - b1 : a1 + b1;
  x2 = S < 0 ? a2 + b2 : a2 - b2;
  x3 = S < 0 ? a2 - b2 : a2 + b2;
}
template <int S>
GL_HD void dft5(g2* x) {
  dft5_part<S>(x[0].re, x[1].re, x[2].re, x[3].re, x[4].re);
  dft5_part<S>(x[0].im, x[1].im, x[2].im, x[3].im, x[4].im);
}

template <int S>
GL_HD void dft7_part(int64_t& x0, int64_t& x1, int64_t& x2, int64_t& x3, int64_t& x4, int64_t& x5, int64_t& x6) {
  constexpr Limbs c1 = k7c1, c2 = k7c2, c3 = k7c3, s1 = k7s1, s2 = k7s2, s3 = k7s3, n1 = k7n1, n3 = k7n3;
  const int64_t p1 = x1 + x6, m1 = x1 - x6, p2 = x2 + x5, m2 = x2 - x5, p3 = x3 + x4, m3 = x3 - x4;
  const int64_t a1 = red(x0 + rdot(p1, c1, p2, c2) + rmul(p3, c3));
  const int64_t a2 = red(x0 + rdot(p1, c2, p2, c3) + rmul(p3, c1));
  const int64_t a3 = red(x0 + rdot(p1, c3, p2, c1) + rmul(p3, c2));
  const int64_t b1 = red(rdot(m1, s1, m2, s2) + rmul(m3, s3));
  const int64_t b2 = red(rdot(m1, s2, m2, n3) + rmul(m3, n1));
  const int64_t b3 = red(rdot(m1, s3, m2, n1) + rmul(m3, s2));
  x0 += red(p1 + p2) + red(p3);
  x1 = S < 0 ? a1 + b1 : a1 - b1;
  x6 = S < 0 ? a1 - b1 : a1 + b1;
  x2 = S < 0 ? a2 + b2 : a2 - b2;
  x5 = S < 0 ? a2 - b2 : a2 + b2;
  x3 = S < 0 ? a3 + b3 : a3 - b3;
  x4 = S < 0 ? a3 - b3 : a3 + b3;
}
template <int S>
GL_HD void dft7(g2* x) {
  dft7_part<S>(x[0].re, x[1].re, x[2].re, x[3].re, x[4].re, x[5].re, x[6].re);
#ifdef __CUDA_ARCH__
  // the imaginary parts after the real ones (no instruction; side by side they spill)
  asm volatile("" : "+l"(x[0].re), "+l"(x[3].re), "+l"(x[1].im), "+l"(x[2].im), "+l"(x[3].im));
#endif
  dft7_part<S>(x[0].im, x[1].im, x[2].im, x[3].im, x[4].im, x[5].im, x[6].im);
}

template <int R, int S>
GL_HD void dft(g2* x) {
  if constexpr (R == 2) dft2<S>(x);
  else if constexpr (R == 3) dft3<S>(x);
  else if constexpr (R == 4) dft4<S>(x);
  else if constexpr (R == 5) dft5<S>(x);
  else dft7<S>(x);
}

// One butterfly of a Stockham stage: v = DFT_R of in(q) w^q; slot(q - 1) is w^q in the
// table of this direction.  Inputs within 3R (first stage: within R, no twiddles), outputs
// 3R.  Radix 8 finishes the even inputs before it reads the odd ones, so that fewer values
// are live at once (80 registers, three CTAs of 256 threads per SM).
template <int R, int S, typename In, typename Slot>
GL_HD void butterfly(g2* v, bool twiddled, const In& in, const Slot& slot) {
  if constexpr (R == 8) {
    if (twiddled) {
      v[0] = red(in(0));
#pragma unroll
      for (int q = 2; q < 8; q += 2) v[q] = cmul(in(q), slot(q - 1));
    } else {
#pragma unroll
      for (int q = 0; q < 8; q += 2) v[q] = in(q);
    }
    dft4_red<S>(v[0], v[2], v[4], v[6]);
    if (twiddled) {
#pragma unroll
      for (int q = 1; q < 8; q += 2) v[q] = cmul(in(q), slot(q - 1));
    } else {
#pragma unroll
      for (int q = 1; q < 8; q += 2) v[q] = in(q);
    }
    dft4_red<S>(v[1], v[3], v[5], v[7]);
    dft8_join<S>(v);
  } else {
    if (twiddled) {
      v[0] = red(in(0));
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = cmul(in(q), slot(q - 1));
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = in(q);
    }
    dft<R, S>(v);
  }
}

// Real-signal split and square for the frequencies k and q k mod M (x^q is conjugation):
// V_k = U_k^2 + c_k D^2, V_qk = U_qk^2 + conj(c_k D^2), D = U_k - conj(U_qk),
// c_k = -(1 + w_M^k)/4.  Inputs within 3R, outputs within R.
GL_HD g2 square(g2 u) {  // within 3R -> within 2R
  const int64_t s = red(u.re + u.im), d = red(u.re - u.im);
  const int64_t r = red(u.re), i = red(u.im);
  return g2{vmul(s, d), vmul(2 * r, i)};
}
GL_HD void pair_square(g2 u, g2 up, int4 c, g2* vk, g2* vkp) {
  const int64_t dr = red(u.re - up.re), di = red(u.im + up.im);
  g2 pc = cmul(g2{vmul(dr + di, red(dr - di)), vmul(2 * dr, di)}, c);
#ifdef __CUDA_ARCH__
  // the squares after the product: computing them side by side takes more registers than
  // four or five resident CTAs leave
  asm("" : "+l"(u.re), "+l"(u.im), "+l"(up.re), "+l"(up.im), "+l"(pc.re), "+l"(pc.im));
#endif
  const g2 s = square(u);
  *vk = red(add(s, pc));
  const g2 sp = square(up);
  *vkp = red(g2{sp.re + pc.re, sp.im - pc.im});
}

// A value within R as two balanced limbs per part, the form of a twiddle: |c0| <= 2^30,
// |c1| <= 2^29 + 16.
GL_HD int4 as_limbs(g2 y) {
  const uint32_t r = lo32((uint64_t)y.re), i = lo32((uint64_t)y.im);
  return make_int4((int)(r << 1) >> 1, limb1(y.re) + (int)((r >> 30) & 1), (int)(i << 1) >> 1,
                   limb1(y.im) + (int)((i >> 30) & 1));
}
GL_HD int4 conj(int4 w) { return make_int4(w.x, w.y, -w.z, -w.w); }

// Biased accumulators of a sum of products of values in limbs.  A product adds at most
// 3 2^60 to lo and 2^61 to mid, so two fit between folds (or one counted twice).
struct Acc {
  uint64_t rl, rm, il, im;
};
GL_HD Acc acc0() { return Acc{kAccLo, kAccMid, kAccLo, kAccMid}; }
GL_HD void acc_mul(Acc& s, int4 x, int4 y) {
  const int c2 = y.y * 2, d2 = y.w * 2, n0 = -y.z, n1 = -y.w, n2 = -d2;
  s.rl = mad_s(x.w, n2, mad_s(x.z, n0, mad_s(x.y, c2, mad_s(x.x, y.x, s.rl))));
  s.rm = mad_s(x.w, n0, mad_s(x.z, n1, mad_s(x.y, y.x, mad_s(x.x, y.y, s.rm))));
  s.il = mad_s(x.w, c2, mad_s(x.z, y.x, mad_s(x.y, d2, mad_s(x.x, y.z, s.il))));
  s.im = mad_s(x.w, y.x, mad_s(x.z, y.y, mad_s(x.y, y.z, mad_s(x.x, y.w, s.im))));
}
GL_HD g2 acc_fold(const Acc& s) { return g2{fold(s.rl, s.rm), fold(s.il, s.im)}; }

// Coefficient b of u(y)^2 mod y^t - z; get(i) is coefficient i of u in limbs.  Within R.
// The products u_i u_j of each half (i + j = b, and i + j = b + t times z) are summed over
// i < j, folded two at a time, and doubled.
template <typename Get>
GL_HD g2 poly_square(const Get& get, int t, int b, int4 z) {
  g2 out = {0, 0};
#pragma unroll 1
  for (int h = b < t - 1 ? 1 : 0; h >= 0; --h) {
    const int s = b + h * t;  // i + j
    int i = h ? b + 1 : 0, j = s - i;
    g2 sum = {0, 0};
#pragma unroll 1
    for (; i + 1 < j - 1; i += 2, j -= 2) {
      Acc a = acc0();
      acc_mul(a, get(i), get(j));
      acc_mul(a, get(i + 1), get(j - 1));
      sum = red(add(sum, acc_fold(a)));
    }
    if (i < j) {
      Acc a = acc0();
      acc_mul(a, get(i), get(j));
      sum = red(add(sum, acc_fold(a)));
      ++i, --j;
    }
    sum = add(sum, sum);
    if (i == j) {
      Acc a = acc0();
      const int4 x = get(i);
      acc_mul(a, x, x);
      sum = add(sum, acc_fold(a));
    }
    out = h ? cmul(red(sum), z) : red(add(out, red(sum)));
  }
  return out;
}
constexpr Limbs kMinusQuarter = limbs(kQ - (1ull << 59));

// v 2^e within R, 0 <= e <= 60: v 2^e = (v >> (61 - e)) 2^61 + the low 61 bits
GL_HD int64_t weighted(int v, int e) {
  const uint64_t x = ((uint64_t)(int64_t)v << e) & kQ;
  const int s = 61 - e;
  return red((int64_t)mad_s(v >> (s < 31 ? s : 31), 1, x));
}

// The integer congruent to x 2^-e in [-2^60 - 4, 2^60 + 3], x within 3R, 0 <= e <= 60.  A
// product of at most kMaxProduct in magnitude is that integer itself: its other
// representatives, q away, lie outside.
constexpr int64_t kMaxProduct = (1ll << 60) - 6;
GL_HD int64_t unweighted(int64_t x, int e) {
  return red((int64_t)(((uint64_t)x << (61 - e)) & kQ) + (x >> e));
}

}  // namespace gf
}  // namespace gl
